// Memory-bound kernels: RMSNorm (+residual) fwd/bwd, SwiGLU fwd/bwd, fused per-head RMSNorm + rotary embedding
// fwd/bwd, KV-cache scatter, AdamW on a flat shard, column-sum reduction.  All use 16-byte vector accesses and
// fp32 math; grids are sized from the row count (one CTA per row, or a persistent multiple of the SM count for
// kernels that also accumulate a per-column reduction).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "rope.cuh"
#include "launch.h"
#include "debug.cuh"
#include "pdl.cuh"

namespace mb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = (threadIdx.x < THREADS / 32) ? sh[threadIdx.x] : 0.f;
  if (w == 0) {
    r = warp_sum(r);
    if (l == 0) sh[0] = r;
  }
  __syncthreads();
  return sh[0];
}

// Copies are one 16-byte access: the members' own copy operators are 4-byte ones, which the compiler does not always join.
struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
  bf16x8() = default;
  __device__ __forceinline__ bf16x8(const bf16x8& o) { *this = o; }
  __device__ __forceinline__ bf16x8& operator=(const bf16x8& o) {
    *reinterpret_cast<uint4*>(this) = *reinterpret_cast<const uint4*>(&o);
    return *this;
  }
};

__device__ __forceinline__ void decode8(const bf16x8& t, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = __bfloat1622float2(t.v[i]);
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const bf16x8 t = *reinterpret_cast<const bf16x8*>(p);
  decode8(t, f);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  bf16x8 t;
#pragma unroll
  for (int i = 0; i < 4; ++i) t.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<bf16x8*>(p) = t;
}

// ---------------------------------------------------------------------------------------------
// RMSNorm forward (optionally fused with the residual add).  H must be a multiple of 8.
//   ADD: r_new = x + residual (rounded to bf16, written to `res_out`), y = rmsnorm(r_new)·w
// ---------------------------------------------------------------------------------------------
// A CTA of ⌈H / (16·N)⌉ threads, whole warps, per row: each has its N 16-byte pieces of either operand in flight at once and keeps the sum as packed bf16; one
// barrier.  The number of threads goes by the width alone, so a token's norm does not depend on how many tokens are beside it.  What bounds it: memory.  Few
// pieces per thread and many small CTAs keep loads, sums and stores of different rows going side by side; a warp per row with all of its pieces, or 256 threads
// with room for 8192 columns and three barriers, went through them in turn.  With the add, µs before → now (at the memory's speed): 7258 rows of 2048
// 31.3 → 19.8 (18.1), 17 829 rows of 1024 35.0 → 24.6 (22.3), of 2048 67.8 → 44.6 (44.6), of 2560 85.4 → 55.3 (55.7), of 4096 142 → 87 (89); one, three or
// four pieces: the same or up to 1 µs slower; with 4-byte accesses (bf16x8) 24.2, 29.3, 54.2, 66.7, 104.
template <bool ADD, int N>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* residual,
                                                          const __nv_bfloat16* __restrict__ w, __nv_bfloat16* y,
                                                          __nv_bfloat16* res_out, float* rstd_out, int H,
                                                          float eps) {
  __shared__ float sh[8];
  pdl_trigger();
  pdl_wait();
  const long long at = blockIdx.x * static_cast<long long>(H);
  const int nvec = H / 8, nt = blockDim.x;
  bf16x8 v[N], r[N];   // all of them requested before the first store: to the compiler the sum may lie over either
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int c = threadIdx.x + nt * i;
    if (c < nvec) {
      v[i] = *reinterpret_cast<const bf16x8*>(x + at + c * 8);
      if (ADD) r[i] = *reinterpret_cast<const bf16x8*>(residual + at + c * 8);
    }
  }
  float ss = 0.f;
  auto take = [&](bf16x8& a, const bf16x8& b, int c) {   // a += b, stored; its squares
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (ADD) {
        const float2 p = __bfloat1622float2(a.v[j]), q = __bfloat1622float2(b.v[j]);
        a.v[j] = __floats2bfloat162_rn(p.x + q.x, p.y + q.y);
      }
      const float2 f = __bfloat1622float2(a.v[j]);
      ss += f.x * f.x + f.y * f.y;
    }
    if (ADD) *reinterpret_cast<bf16x8*>(res_out + at + c * 8) = a;
  };
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (threadIdx.x + nt * i < nvec) take(v[i], r[i], threadIdx.x + nt * i);
  for (int c = threadIdx.x + N * nt; c < nvec; c += nt) {   // rows beyond 8192 columns: read again from L2
    bf16x8 a = *reinterpret_cast<const bf16x8*>(x + at + c * 8), b = a;
    if (ADD) b = *reinterpret_cast<const bf16x8*>(residual + at + c * 8);
    take(a, b, c);
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i < nt / 32) ss += sh[i];
  const float rstd = rsqrtf(ss / H + eps);
  if (threadIdx.x == 0 && rstd_out != nullptr) rstd_out[blockIdx.x] = rstd;
  auto put = [&](const bf16x8& a, int c) {
    const bf16x8 wv = *reinterpret_cast<const bf16x8*>(w + c * 8);
    bf16x8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(a.v[j]), g = __bfloat1622float2(wv.v[j]);
      o.v[j] = __floats2bfloat162_rn(f.x * rstd * g.x, f.y * rstd * g.y);
    }
    *reinterpret_cast<bf16x8*>(y + at + c * 8) = o;
  };
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (threadIdx.x + nt * i < nvec) put(v[i], threadIdx.x + nt * i);
  for (int c = threadIdx.x + N * nt; c < nvec; c += nt) put(*reinterpret_cast<const bf16x8*>((ADD ? res_out : x) + at + c * 8), c);
}

// RMSNorm backward.  x is the normalised input (the post-add residual stream), dy the gradient of y,
// `dres` an optional extra gradient flowing into x directly (the residual branch).
//   dx = rstd·(w·dy − x̂·mean(w·dy·x̂)) + dres ;   dw_partial[block] += dy·x̂
// Persistent grid; each CTA writes one row of fp32 partial dw sums, reduced by `colsum_kernel`.
__global__ void __launch_bounds__(256) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                          const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ dres,
                                                          const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                                                          float* __restrict__ dw_partial, int T, int H) {
  __shared__ float sh[32];
  constexpr int MAXI = 4;
  const int nvec = H / 8;
  float dwacc[MAXI][8];
#pragma unroll
  for (int it = 0; it < MAXI; ++it)
#pragma unroll
    for (int i = 0; i < 8; ++i) dwacc[it][i] = 0.f;
  for (long long row = blockIdx.x; row < T; row += gridDim.x) {
    const float rstd = rstd_in[row];
    float xh[MAXI][8], g[MAXI][8];
    float dot = 0.f;
#pragma unroll
    for (int it = 0; it < MAXI; ++it) {
      const int v = threadIdx.x + it * 256;
      if (v < nvec) {
        float xv[8], dv[8], wv[8];
        load8(x + row * H + v * 8, xv);
        load8(dy + row * H + v * 8, dv);
        load8(w + v * 8, wv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xh[it][i] = xv[i] * rstd;
          g[it][i] = dv[i] * wv[i];
          dot += g[it][i] * xh[it][i];
          dwacc[it][i] += dv[i] * xh[it][i];
        }
      }
    }
    dot = block_sum<256>(dot, sh) / H;
#pragma unroll
    for (int it = 0; it < MAXI; ++it) {
      const int v = threadIdx.x + it * 256;
      if (v < nvec) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = rstd * (g[it][i] - xh[it][i] * dot);
        if (dres != nullptr) {
          float r[8];
          load8(dres + row * H + v * 8, r);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += r[i];
        }
        store8(dx + row * H + v * 8, o);
      }
    }
  }
#pragma unroll
  for (int it = 0; it < MAXI; ++it) {
    const int v = threadIdx.x + it * 256;
    if (v < nvec) {
#pragma unroll
      for (int i = 0; i < 8; ++i) dw_partial[static_cast<long long>(blockIdx.x) * H + v * 8 + i] = dwacc[it][i];
    }
  }
}

// The same with WPR warps per row, for rows of 256·VPL·WPR elements: all loads of a row in flight at once and no CTA barrier per row (the form
// above waits for two of them: 98 µs at 12 075 × 2048 where the bytes take 31).  VPL is kept at 5 or below: the row, its gradient
// and the weight gradient's sums have to fit the registers of 12 (VPL 5: 8) warps per SM.  The sums stay in registers until the end, where the
// CTA's warps add theirs up in shared memory.  The residual's gradient is requested with the row: behind the sums it was a second trip to memory per
// row (12 075 × 2048 69 → 44 µs, 11 791 × 2560 99 → 53; 30 and 37 at the memory's speed).
template <int VPL, int WPR>
__global__ void __launch_bounds__(128, VPL <= 4 ? 3 : 2) rmsnorm_bwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                  const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ dres,
                                                                  const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                                                                  float* __restrict__ dw_partial, int T) {
  constexpr int H = VPL * WPR * 256, kGroups = 4 / WPR, kStep = 32 * WPR;
  __shared__ float sh_dw[kGroups][H];
  __shared__ float sh_dot[2][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = warp / WPR, v0 = (warp % WPR) * 32 + lane;
  float dwacc[VPL][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
  int parity = 0;
  for (long long row = static_cast<long long>(blockIdx.x) * kGroups + group; row < T; row += static_cast<long long>(gridDim.x) * kGroups) {
    const float rstd = rstd_in[row];
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * H) + v0;
    const bf16x8* gr = reinterpret_cast<const bf16x8*>(dy + row * H) + v0;
    const bf16x8* wr = reinterpret_cast<const bf16x8*>(w) + v0;
    bf16x8 xv[VPL], gv[VPL], rv[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      xv[i] = xr[kStep * i];
      gv[i] = gr[kStep * i];
      if (dres != nullptr) rv[i] = (reinterpret_cast<const bf16x8*>(dres + row * H) + v0)[kStep * i];
    }
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const bf16x8 wv = wr[kStep * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = __bfloat1622float2(xv[i].v[j]), g = __bfloat1622float2(gv[i].v[j]), c = __bfloat1622float2(wv.v[j]);
        const float x0 = a.x * rstd, x1 = a.y * rstd;
        dot += g.x * c.x * x0;
        dot += g.y * c.y * x1;
        dwacc[i][2 * j] += g.x * x0;
        dwacc[i][2 * j + 1] += g.y * x1;
      }
    }
    dot = warp_sum(dot);
    if (WPR > 1) {                         // the row's warps exchange their sums; two buffers, so one barrier per row is enough
      if (lane == 0) sh_dot[parity][warp] = dot;
      asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(32 * WPR) : "memory");
      dot = 0.f;
#pragma unroll
      for (int k = 0; k < WPR; ++k) dot += sh_dot[parity][group * WPR + k];
      parity ^= 1;
    }
    dot /= H;
    // the row is decoded again from its 16-bit form: kept decoded it would not fit the registers
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm volatile("" : "+r"(reinterpret_cast<uint32_t&>(xv[i].v[j])), "+r"(reinterpret_cast<uint32_t&>(gv[i].v[j])));
    bf16x8* dr = reinterpret_cast<bf16x8*>(dx + row * H) + v0;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const bf16x8 wv = wr[kStep * i];
      bf16x8 o;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = __bfloat1622float2(xv[i].v[j]), g = __bfloat1622float2(gv[i].v[j]), c = __bfloat1622float2(wv.v[j]);
        float o0 = rstd * (g.x * c.x - a.x * rstd * dot), o1 = rstd * (g.y * c.y - a.y * rstd * dot);
        if (dres != nullptr) {
          const float2 r = __bfloat1622float2(rv[i].v[j]);
          o0 += r.x;
          o1 += r.y;
        }
        o.v[j] = __floats2bfloat162_rn(o0, o1);
      }
      dr[kStep * i] = o;
    }
  }
#pragma unroll
  for (int i = 0; i < VPL; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) sh_dw[group][(v0 + kStep * i) * 8 + j] = dwacc[i][j];
  __syncthreads();
  for (int c = threadIdx.x; c < H; c += 128) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kGroups; ++k) s += sh_dw[k][c];
    dw_partial[static_cast<long long>(blockIdx.x) * H + c] = s;
  }
}

// out[c] = Σ_r partial[r, c]  (fp32 in, bf16 or fp32 out).  32 columns per CTA, the rows dealt to its 32 warps: one thread per column waits
// for up to 592 loads in a row (28.6 µs at 592 × 2560; 4.7 this way).
__global__ void __launch_bounds__(1024) colsum_kernel(const float* __restrict__ partial, void* __restrict__ out, int R, int C, int out_fp32) {
  __shared__ float sh[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < C) {
#pragma unroll 8
    for (int r = warp; r < R; r += 32) s += partial[static_cast<long long>(r) * C + c];
  }
  sh[warp][lane] = s;
  __syncthreads();
  s = warp_sum(sh[lane][warp]);            // warp w adds up column w
  if (lane == 0 && blockIdx.x * 32 + warp < C) {
    if (out_fp32) reinterpret_cast<float*>(out)[blockIdx.x * 32 + warp] = s;
    else reinterpret_cast<__nv_bfloat16*>(out)[blockIdx.x * 32 + warp] = __float2bfloat16(s);
  }
}

// ---------------------------------------------------------------------------------------------
// SwiGLU: in [T, 2F] (gate | up) → out [T, F].  11 791 rows of 9728 107 → 102 µs with an item per thread (`item_grid`; 105 at the copy rate)
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const __nv_bfloat16* in, __nv_bfloat16* out,
                                                         long long T, int F, const int* rows_ptr) {
  pdl_trigger();
  pdl_wait();
  const int nvec = F / 8;
  if (rows_ptr != nullptr) T = min(T, static_cast<long long>(*rows_ptr));  // device-side row count (MoE padded buffers)
  const long long total = T * nvec;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * 256) {
    const long long t = i / nvec;
    const int v = static_cast<int>(i % nvec);
    float g[8], u[8], o[8];
    load8(in + t * 2 * F + v * 8, g);
    load8(in + t * 2 * F + F + v * 8, u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = g[k] / (1.f + __expf(-g[k])) * u[k];
    store8(out + t * F + v * 8, o);
  }
}

// act (null, or in dout's place): the activation itself, for the gradient of the weight behind it.  Read once instead of twice.  11 791 rows of 9728:
// 156 + 252 µs in two kernels, 279 in one; 201 with 16-byte accesses (232) and an item per thread (`item_grid`).
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ in, const __nv_bfloat16* dout,
                                                         __nv_bfloat16* __restrict__ din, __nv_bfloat16* act, long long T, int F,
                                                         const int* __restrict__ rows_ptr) {
  const int nvec = F / 8;
  if (rows_ptr != nullptr) T = min(T, static_cast<long long>(*rows_ptr));
  const long long total = T * nvec;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * 256) {
    const long long t = i / nvec;
    const int v = static_cast<int>(i % nvec);
    float g[8], u[8], d[8], dg[8], du[8];
    load8(in + t * 2 * F + v * 8, g);
    load8(in + t * 2 * F + F + v * 8, u);
    load8(dout + t * F + v * 8, d);
    if (act != nullptr) {
      float a[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] = g[k] / (1.f + __expf(-g[k])) * u[k];
      store8(act + t * F + v * 8, a);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float s = 1.f / (1.f + __expf(-g[k]));
      dg[k] = d[k] * u[k] * s * (1.f + g[k] * (1.f - s));
      du[k] = d[k] * g[k] * s;
    }
    store8(din + t * 2 * F + v * 8, dg);
    store8(din + t * 2 * F + F + v * 8, du);
  }
}

// ---------------------------------------------------------------------------------------------
// Per-head RMSNorm (optional) + NeoX rotary embedding on q and k, in one pass.  One warp per (token, head).
// Layout [T, heads, D]; pairs are (i, i + D/2).  D ∈ {64, 128}.
// ---------------------------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void norm_rope_row(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                              const __nv_bfloat16* __restrict__ w, float pos, float log2_theta, float eps,
                                              float* rstd_out, int lane, __nv_bfloat16* __restrict__ dst2 = nullptr) {
  constexpr int EPL = D / 64;  // elements per lane in each half
  __nv_bfloat16 o1[EPL], o2[EPL];
  norm_rope_values<D>(src, w, pos, log2_theta, eps, rstd_out, lane, o1, o2);
#pragma unroll
  for (int e = 0; e < EPL; ++e) {
    const int j = lane * EPL + e;
    dst[j] = o1[e];
    dst[D / 2 + j] = o2[e];
    if (dst2 != nullptr) {
      dst2[j] = o1[e];
      dst2[D / 2 + j] = o2[e];
    }
  }
}

// Many tokens, D = 128: four heads of a token per warp, sixteen lanes per head with 8-byte pieces of both halves; all loads of the warp go out
// together and the angles are computed once for two heads.  One warp per head is bound by instructions (2-byte loads, the angles
// 40 times per token).  7258 tokens × 40 heads with the cache 67.5 → 40.5 µs, 11 791 × 40 without 122 → 71 µs (37 at the memory's speed).
__global__ void __launch_bounds__(256) qk_norm_rope_many_kernel(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                                                                long long q_tok_stride, long long k_tok_stride, long long v_tok_stride,
                                                                const __nv_bfloat16* qw, const __nv_bfloat16* kw, const int* positions,
                                                                __nv_bfloat16* qo, __nv_bfloat16* ko, float* q_rstd, float* k_rstd,
                                                                __nv_bfloat16* kc, __nv_bfloat16* vc, const long long* slots, long long T, int Hq,
                                                                int Hk, float log2_theta, float eps) {
  constexpr int D = 128;
  typedef __nv_bfloat16 bf;
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, half = lane >> 4, j = (lane & 15) * 4;
  const int quads = (Hq + (vc != nullptr ? 2 : 1) * Hk) / 4;
  const long long wid = (blockIdx.x * 256ll + threadIdx.x) >> 5;
  if (wid >= T * quads) return;
  const long long t = wid / quads;
  const int h = static_cast<int>(wid % quads) * 4;             // first head of the four: all of q, all of k or all of v
  long long slot = slots != nullptr && h >= Hq ? slots[t] : -1;
  if (slot >= 0 && !dbg::in_bounds(dbg::kKvSlots, slot, 101)) slot = -1;   // debug build: a slot outside the cache is recorded, not written
  const bool is_q = h < Hq, is_v = h >= Hq + Hk;
  const bf* src = is_q ? q + t * q_tok_stride + h * D : is_v ? v + t * v_tok_stride + (h - Hq - Hk) * D : k + t * k_tok_stride + (h - Hq) * D;
  uint2 a[2], b[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    a[i] = *reinterpret_cast<const uint2*>(src + (2 * i + half) * D + j);
    b[i] = *reinterpret_cast<const uint2*>(src + (2 * i + half) * D + D / 2 + j);
  }
  bf* cached = is_v ? vc + (slot * Hk + h - Hq - Hk) * D : kc + (slot * Hk + h - Hq) * D;    // used where slot >= 0
  if (is_v) {
    if (slot < 0) return;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      *reinterpret_cast<uint2*>(cached + (2 * i + half) * D + j) = a[i];
      *reinterpret_cast<uint2*>(cached + (2 * i + half) * D + D / 2 + j) = b[i];
    }
    return;
  }
  const bf* w = is_q ? qw : kw;
  float wa[4], wb[4], sn[4], cs[4];
  const float pos = static_cast<float>(positions[t]);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    wa[e] = w != nullptr ? __bfloat162float(w[j + e]) : 1.f;
    wb[e] = w != nullptr ? __bfloat162float(w[D / 2 + j + e]) : 1.f;
    sincosf(pos * exp2f(-log2_theta * (2.f * (j + e)) / D), &sn[e], &cs[e]);
  }
  bf* dst = is_q ? qo + (t * Hq + h) * D : ko + (t * Hk + h - Hq) * D;
  float* rstd_out = is_q ? (q_rstd != nullptr ? q_rstd + t * Hq + h : nullptr) : (k_rstd != nullptr ? k_rstd + t * Hk + h - Hq : nullptr);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bf *pa = reinterpret_cast<const bf*>(&a[i]), *pb = reinterpret_cast<const bf*>(&b[i]);
    float x1[4], x2[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x1[e] = __bfloat162float(pa[e]);
      x2[e] = __bfloat162float(pb[e]);
    }
    if (w != nullptr) {
      // the order of norm_rope_row's sum, so that a token is normed alike in every batch: its lanes 2l and 2l + 1 hold what is this lane's,
      // and meet in the last step
      float ss[2] = {0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 4; ++e) ss[e >> 1] += x1[e] * x1[e] + x2[e] * x2[e];
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) {
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], d);
        ss[1] += __shfl_xor_sync(0xffffffffu, ss[1], d);
      }
      const float rstd = rsqrtf((ss[0] + ss[1]) / D + eps);
      if (rstd_out != nullptr && (lane & 15) == 0) rstd_out[2 * i + half] = rstd;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x1[e] = __bfloat162float(__float2bfloat16(x1[e] * rstd * wa[e]));
        x2[e] = __bfloat162float(__float2bfloat16(x2[e] * rstd * wb[e]));
      }
    }
    uint2 o1, o2;
    bf *p1 = reinterpret_cast<bf*>(&o1), *p2 = reinterpret_cast<bf*>(&o2);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 r = rotate_pair(x1[e], x2[e], cs[e], sn[e]);
      p1[e] = __float2bfloat16(r.x);
      p2[e] = __float2bfloat16(r.y);
    }
    bf* to = dst + (2 * i + half) * D + j;
    *reinterpret_cast<uint2*>(to) = o1;
    *reinterpret_cast<uint2*>(to + D / 2) = o2;
    if (slot >= 0) {
      bf* to2 = cached + (2 * i + half) * D + j;
      *reinterpret_cast<uint2*>(to2) = o1;
      *reinterpret_cast<uint2*>(to2 + D / 2) = o2;
    }
  }
}

// From where four heads per warp fill the chip (148 SMs × 16 warps), if no warp has heads of two tensors and all pieces are aligned.
static bool rope_by_fours(long long T, int Hq, int Hk, int heads, int D, long long strides, uintptr_t pointers) {
  return D == 128 && Hq % 4 == 0 && Hk % 4 == 0 && T * (heads / 4) >= 148 * 16 && (strides & 3) == 0 && (pointers & 7) == 0;
}

// Engine form: the same per-head norm + rotary for q and k, with the rotated k and the raw v also written into the
// paged KV cache at each token's slot (slot < 0: token not cached).  One warp per (token, q/k/v head).
template <int D>
__global__ void __launch_bounds__(256) qk_norm_rope_cache_kernel(const __nv_bfloat16* q, const __nv_bfloat16* k,
                                                                 const __nv_bfloat16* v, long long q_tok_stride,
                                                                 long long k_tok_stride, long long v_tok_stride,
                                                                 const __nv_bfloat16* __restrict__ qw, const __nv_bfloat16* __restrict__ kw,
                                                                 const int* positions, __nv_bfloat16* qo,
                                                                 __nv_bfloat16* ko, __nv_bfloat16* kc,
                                                                 __nv_bfloat16* vc, const long long* slots,
                                                                 long long T, int Hq, int Hk, float log2_theta, float eps) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long wid = (blockIdx.x * 256ll + threadIdx.x) >> 5;
  const int heads = Hq + 2 * Hk;
  if (wid >= T * heads) return;
  const long long t = wid / heads;
  const int h = static_cast<int>(wid % heads);
  if (h < Hq) {
    norm_rope_row<D>(q + t * q_tok_stride + h * D, qo + (t * Hq + h) * D, qw, static_cast<float>(positions[t]), log2_theta, eps,
                     nullptr, lane);
    return;
  }
  long long slot = slots[t];
  if (slot >= 0 && !dbg::in_bounds(dbg::kKvSlots, slot, 101)) slot = -1;   // debug build: a slot outside the cache is recorded, not written
  if (h < Hq + Hk) {
    const int hk = h - Hq;
    norm_rope_row<D>(k + t * k_tok_stride + hk * D, ko + (t * Hk + hk) * D, kw, static_cast<float>(positions[t]), log2_theta, eps,
                     nullptr, lane, slot >= 0 ? kc + (slot * Hk + hk) * D : nullptr);
  } else if (slot >= 0) {
    const int hk = h - Hq - Hk;
    constexpr int EPL = D / 32;   // 4 (8 bytes) or 2 (4 bytes) elements per lane
    const __nv_bfloat16* src = v + t * v_tok_stride + hk * D + lane * EPL;
    __nv_bfloat16* dst = vc + (slot * Hk + hk) * D + lane * EPL;
    if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) % (2 * EPL)) {   // rows of a view that starts anywhere
#pragma unroll
      for (int e = 0; e < EPL; ++e) dst[e] = src[e];
    } else if (EPL == 4) {
      *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(src);
    } else {
      *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(src);
    }
  }
}

template <int D>
__global__ void __launch_bounds__(256) qk_norm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                               long long q_tok_stride, long long k_tok_stride,
                                                               const __nv_bfloat16* __restrict__ qw, const __nv_bfloat16* __restrict__ kw,
                                                               const int* __restrict__ positions, __nv_bfloat16* __restrict__ qo,
                                                               __nv_bfloat16* __restrict__ ko, float* __restrict__ q_rstd,
                                                               float* __restrict__ k_rstd, long long T, int Hq, int Hk, float log2_theta,
                                                               float eps) {
  const int lane = threadIdx.x & 31;
  const long long wid = (blockIdx.x * 256ll + threadIdx.x) >> 5;
  const int heads = Hq + Hk;
  if (wid >= T * heads) return;
  const long long t = wid / heads;
  const int h = static_cast<int>(wid % heads);
  const float pos = static_cast<float>(positions[t]);
  if (h < Hq) {
    norm_rope_row<D>(q + t * q_tok_stride + h * D, qo + (t * Hq + h) * D, qw, pos, log2_theta, eps,
                     q_rstd ? q_rstd + t * Hq + h : nullptr, lane);
  } else {
    const int hk = h - Hq;
    norm_rope_row<D>(k + t * k_tok_stride + hk * D, ko + (t * Hk + hk) * D, kw, pos, log2_theta, eps,
                     k_rstd ? k_rstd + t * Hk + hk : nullptr, lane);
  }
}

// Backward: un-rotate the incoming gradient, then the RMSNorm backward per head.  dw partial sums per CTA.
template <int D>
__global__ void __launch_bounds__(256) qk_norm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ x, long long x_tok_stride,
                                                               const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                                                               const __nv_bfloat16* __restrict__ dy, const int* __restrict__ positions,
                                                               __nv_bfloat16* __restrict__ dx, long long dx_tok_stride,
                                                               float* __restrict__ dw_partial, long long T, int Hn, float log2_theta) {
  constexpr int EPL = D / 64;
  __shared__ float sh_dw[8][D];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float dwa[EPL], dwb[EPL];
#pragma unroll
  for (int e = 0; e < EPL; ++e) dwa[e] = dwb[e] = 0.f;
  // a warp takes four heads of a token: their angles are computed once and the heads' loads are in flight together
  constexpr int HPW = 4;
  const int parts = (Hn + HPW - 1) / HPW;
  const long long items = T * parts;
  for (long long it = (blockIdx.x * 256ll + threadIdx.x) >> 5; it < items; it += (static_cast<long long>(gridDim.x) * 256) >> 5) {
    const long long t = it / parts;
    const int h0 = static_cast<int>(it % parts) * HPW;
    const float pos = static_cast<float>(positions[t]);
    float sn[EPL], cs[EPL];
#pragma unroll
    for (int e = 0; e < EPL; ++e) sincosf(pos * exp2f(-log2_theta * (2.f * (lane * EPL + e)) / D), &sn[e], &cs[e]);
    __nv_bfloat16 gl[HPW][2 * EPL], xl[HPW][2 * EPL];
    float rs[HPW];
#pragma unroll
    for (int i = 0; i < HPW; ++i) {
      if (h0 + i >= Hn) break;
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        const __nv_bfloat16* gr = dy + (t * Hn + h0 + i) * D + lane * EPL + e;
        gl[i][e] = gr[0];
        gl[i][EPL + e] = gr[D / 2];
        if (w != nullptr) {
          const __nv_bfloat16* xr = x + t * x_tok_stride + (h0 + i) * D + lane * EPL + e;
          xl[i][e] = xr[0];
          xl[i][EPL + e] = xr[D / 2];
        }
      }
      rs[i] = w != nullptr ? rstd_in[t * Hn + h0 + i] : 1.f;
    }
#pragma unroll
    for (int i = 0; i < HPW; ++i) {
      if (h0 + i >= Hn) break;
      __nv_bfloat16* dr = dx + t * dx_tok_stride + (h0 + i) * D;
      float g1[EPL], g2[EPL];
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        const float d1 = __bfloat162float(gl[i][e]), d2 = __bfloat162float(gl[i][EPL + e]);
        g1[e] = d1 * cs[e] + d2 * sn[e];   // transpose of the rotation
        g2[e] = d2 * cs[e] - d1 * sn[e];
      }
      if (w == nullptr) {
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          dr[lane * EPL + e] = __float2bfloat16(g1[e]);
          dr[D / 2 + lane * EPL + e] = __float2bfloat16(g2[e]);
        }
        continue;
      }
      const float rstd = rs[i];
      float xa[EPL], xb[EPL], ga[EPL], gb[EPL];
      float dot = 0.f;
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        const int j = lane * EPL + e;
        xa[e] = __bfloat162float(xl[i][e]) * rstd;
        xb[e] = __bfloat162float(xl[i][EPL + e]) * rstd;
        ga[e] = g1[e] * __bfloat162float(w[j]);
        gb[e] = g2[e] * __bfloat162float(w[D / 2 + j]);
        dot += ga[e] * xa[e] + gb[e] * xb[e];
        dwa[e] += g1[e] * xa[e];
        dwb[e] += g2[e] * xb[e];
      }
      dot = warp_sum(dot) / D;
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        dr[lane * EPL + e] = __float2bfloat16(rstd * (ga[e] - xa[e] * dot));
        dr[D / 2 + lane * EPL + e] = __float2bfloat16(rstd * (gb[e] - xb[e] * dot));
      }
    }
  }
  if (w != nullptr && dw_partial != nullptr) {
#pragma unroll
    for (int e = 0; e < EPL; ++e) {
      sh_dw[wib][lane * EPL + e] = dwa[e];
      sh_dw[wib][D / 2 + lane * EPL + e] = dwb[e];
    }
    __syncthreads();
    if (threadIdx.x < D) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) s += sh_dw[i][threadIdx.x];
      dw_partial[static_cast<long long>(blockIdx.x) * D + threadIdx.x] = s;
    }
  }
}

// The same for D = 128 with a norm and heads in fours: sixteen lanes per head with 8-byte pieces of both halves, two heads at a time, all loads of the four
// heads together, frequencies and weights in registers.  A warp per head with 2-byte loads was bound by instructions: 11 791 tokens × 32 heads
// 104 → 72 µs (44 at the memory's speed).
__global__ void __launch_bounds__(256) qk_norm_rope_bwd_many_kernel(const __nv_bfloat16* __restrict__ x, long long x_tok_stride,
                                                                    const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                                                                    const __nv_bfloat16* __restrict__ dy, const int* __restrict__ positions,
                                                                    __nv_bfloat16* __restrict__ dx, long long dx_tok_stride,
                                                                    float* __restrict__ dw_partial, long long T, int Hn, float log2_theta) {
  constexpr int D = 128;
  __shared__ float sh_dw[16][D];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, half = lane >> 4, j = (lane & 15) * 4;
  float freq[4], wa[4], wb[4], dwa[4], dwb[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    freq[e] = exp2f(-log2_theta * (2.f * (j + e)) / D);
    wa[e] = __bfloat162float(w[j + e]);
    wb[e] = __bfloat162float(w[D / 2 + j + e]);
    dwa[e] = dwb[e] = 0.f;
  }
  auto four = [](const uint2& v, float (&f)[4]) {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
  };
  auto pack4 = [](const float (&f)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  };
  const int quads = Hn / 4;
  const long long items = T * quads;
  for (long long it = (blockIdx.x * 256ll + threadIdx.x) >> 5; it < items; it += (static_cast<long long>(gridDim.x) * 256) >> 5) {
    const long long t = it / quads;
    const int h0 = static_cast<int>(it % quads) * 4 + half;
    uint2 gl[2][2], xl[2][2];
    float rs[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const __nv_bfloat16* gr = dy + (t * Hn + h0 + 2 * i) * D + j;
      const __nv_bfloat16* xr = x + t * x_tok_stride + (h0 + 2 * i) * D + j;
      gl[i][0] = *reinterpret_cast<const uint2*>(gr);
      gl[i][1] = *reinterpret_cast<const uint2*>(gr + D / 2);
      xl[i][0] = *reinterpret_cast<const uint2*>(xr);
      xl[i][1] = *reinterpret_cast<const uint2*>(xr + D / 2);
      rs[i] = rstd_in[t * Hn + h0 + 2 * i];
    }
    const float pos = static_cast<float>(positions[t]);
    float sn[4], cs[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) sincosf(pos * freq[e], &sn[e], &cs[e]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float d1[4], d2[4], xa[4], xb[4], o1[4], o2[4], dot = 0.f;
      four(gl[i][0], d1);
      four(gl[i][1], d2);
      four(xl[i][0], xa);
      four(xl[i][1], xb);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float g1 = d1[e] * cs[e] + d2[e] * sn[e], g2 = d2[e] * cs[e] - d1[e] * sn[e];     // transpose of the rotation
        xa[e] *= rs[i];
        xb[e] *= rs[i];
        d1[e] = g1 * wa[e];
        d2[e] = g2 * wb[e];
        dot += d1[e] * xa[e] + d2[e] * xb[e];
        dwa[e] += g1 * xa[e];
        dwb[e] += g2 * xb[e];
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      dot /= D;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o1[e] = rs[i] * (d1[e] - xa[e] * dot);
        o2[e] = rs[i] * (d2[e] - xb[e] * dot);
      }
      __nv_bfloat16* dr = dx + t * dx_tok_stride + (h0 + 2 * i) * D + j;
      *reinterpret_cast<uint2*>(dr) = pack4(o1);
      *reinterpret_cast<uint2*>(dr + D / 2) = pack4(o2);
    }
  }
  if (dw_partial == nullptr) return;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    sh_dw[2 * wib + half][j + e] = dwa[e];
    sh_dw[2 * wib + half][D / 2 + j + e] = dwb[e];
  }
  __syncthreads();
  if (threadIdx.x < D) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) s += sh_dw[i][threadIdx.x];
    dw_partial[static_cast<long long>(blockIdx.x) * D + threadIdx.x] = s;
  }
}

// ---------------------------------------------------------------------------------------------
// Rotary embedding alone (NeoX pairing: element i rotates with element i + D/2), forward or inverse (= its own backward).
// One warp per (token, head); x [T, H, D] with token stride `tok_stride`, y contiguous.
// ---------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(256) rope_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                                   const int* __restrict__ positions, long long T, int H, long long tok_stride,
                                                   float log2_theta, int inverse) {
  const int lane = threadIdx.x & 31;
  const long long wid = (blockIdx.x * 256ll + threadIdx.x) >> 5;
  if (wid >= T * H) return;
  const long long t = wid / H;
  const int h = static_cast<int>(wid % H);
  const __nv_bfloat16* src = x + t * tok_stride + static_cast<long long>(h) * D;
  __nv_bfloat16* dst = y + (t * H + h) * D;
  const float pos = static_cast<float>(positions[t]);
  constexpr int HALF = D / 2;
#pragma unroll
  for (int i = lane; i < HALF; i += 32) {
    const float inv_freq = exp2f(-log2_theta * (static_cast<float>(2 * i) / D));
    float sn, cs;
    sincosf(pos * inv_freq, &sn, &cs);
    if (inverse) sn = -sn;
    const float a = __bfloat162float(src[i]), b = __bfloat162float(src[i + HALF]);
    dst[i] = __float2bfloat16(a * cs - b * sn);
    dst[i + HALF] = __float2bfloat16(b * cs + a * sn);
  }
}

// ---------------------------------------------------------------------------------------------
// KV cache scatter: rows [T, Hkv·D] → cache[slot, Hkv·D]
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) kv_cache_write_kernel(const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
                                                             long long k_stride, long long v_stride, __nv_bfloat16* __restrict__ kc,
                                                             __nv_bfloat16* __restrict__ vc, const long long* __restrict__ slots,
                                                             long long T, int row_elems) {
  const int nvec = row_elems / 8;
  const long long total = T * nvec;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * 256) {
    const long long t = i / nvec;
    const int c = static_cast<int>(i % nvec) * 8;
    const long long slot = slots[t];
    if (slot < 0 || !dbg::in_bounds(dbg::kKvSlots, slot, 102)) continue;
    *reinterpret_cast<uint4*>(kc + slot * row_elems + c) = *reinterpret_cast<const uint4*>(k + t * k_stride + c);
    *reinterpret_cast<uint4*>(vc + slot * row_elems + c) = *reinterpret_cast<const uint4*>(v + t * v_stride + c);
  }
}

// ---------------------------------------------------------------------------------------------
// Rows of a paged cache, keys and values of every slot in one launch: cache[slots[t], Hkv·D] → k, v [n, Hkv·D].  A warp has four slots, whose eight pieces
// of 16 bytes per lane are requested together.  A slot outside the cache sets the error flag and gives zeros.  What bounds it: the cache's rows from
// memory (the copies stay in L2 for the attention behind it).  18 000 slots of 4 heads × 128: from the rotation's end to the
// attention's start 19 µs with two index_select launches (8.4 + 8.1), 11 with this one.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) kv_gather_kernel(const __nv_bfloat16* kc, const __nv_bfloat16* vc, const long long* slots, long long n,
                                                        long long n_slots, int row_elems, __nv_bfloat16* k, __nv_bfloat16* v, int* error_flag) {
  constexpr int U = 4;
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, nvec = row_elems / 8;
  const long long t0 = (blockIdx.x * 8ll + (threadIdx.x >> 5)) * U;
  if (t0 >= n) return;
  long long at[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    at[u] = t0 + u < n ? slots[t0 + u] : 0;
    if (at[u] < 0 || at[u] >= n_slots) {
      if (lane == 0) atomicCAS(error_flag, 0, 73);
      at[u] = -1;
    }
  }
  for (int c = lane; c < nvec; c += 32) {
    uint4 kr[U], vr[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      kr[u] = vr[u] = make_uint4(0, 0, 0, 0);
      if (t0 + u < n && at[u] >= 0) {
        kr[u] = *reinterpret_cast<const uint4*>(kc + at[u] * row_elems + c * 8);
        vr[u] = *reinterpret_cast<const uint4*>(vc + at[u] * row_elems + c * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (t0 + u < n) {
        *reinterpret_cast<uint4*>(k + (t0 + u) * row_elems + c * 8) = kr[u];
        *reinterpret_cast<uint4*>(v + (t0 + u) * row_elems + c * 8) = vr[u];
      }
  }
}

// ---------------------------------------------------------------------------------------------
// AdamW on a flat fp32 shard with a per-element decay mask and a device-side gradient scale; writes the
// updated parameter in bf16 (or fp32) to `param_out`.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ master, const float* __restrict__ grad, float* __restrict__ m,
                                                    float* __restrict__ v, const float* __restrict__ decay_mask,
                                                    const float* __restrict__ scale_ptr, void* __restrict__ param_out, int out_bf16,
                                                    long long n, float lr, float b1, float b2, float eps, float wd, float bc1,
                                                    float bc2) {
  const float scale = scale_ptr ? *scale_ptr : 1.f;
  for (long long i = (blockIdx.x * 256ll + threadIdx.x) * 4; i < n; i += static_cast<long long>(gridDim.x) * 256 * 4) {
    if (i + 4 <= n) {
      float4 g = *reinterpret_cast<const float4*>(grad + i);
      float4 mm = *reinterpret_cast<const float4*>(m + i);
      float4 vv = *reinterpret_cast<const float4*>(v + i);
      float4 p = *reinterpret_cast<const float4*>(master + i);
      float4 dm = decay_mask ? *reinterpret_cast<const float4*>(decay_mask + i) : make_float4(1.f, 1.f, 1.f, 1.f);
      float* gp = reinterpret_cast<float*>(&g);
      float* mp = reinterpret_cast<float*>(&mm);
      float* vp = reinterpret_cast<float*>(&vv);
      float* pp = reinterpret_cast<float*>(&p);
      float* dp = reinterpret_cast<float*>(&dm);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float gs = gp[k] * scale;
        mp[k] = b1 * mp[k] + (1.f - b1) * gs;
        vp[k] = b2 * vp[k] + (1.f - b2) * gs * gs;
        const float denom = sqrtf(vp[k] / bc2) + eps;
        pp[k] = pp[k] * (1.f - lr * wd * dp[k]) - lr * (mp[k] / bc1) / denom;
      }
      *reinterpret_cast<float4*>(m + i) = mm;
      *reinterpret_cast<float4*>(v + i) = vv;
      *reinterpret_cast<float4*>(master + i) = p;
      if (param_out != nullptr) {
        if (out_bf16) {
          uint2 o;
          __nv_bfloat162 lo = __floats2bfloat162_rn(pp[0], pp[1]);
          __nv_bfloat162 hi = __floats2bfloat162_rn(pp[2], pp[3]);
          o.x = *reinterpret_cast<uint32_t*>(&lo);
          o.y = *reinterpret_cast<uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(param_out) + i) = o;
        } else {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(param_out) + i) = p;
        }
      }
    } else {
      for (long long j = i; j < n; ++j) {
        const float gs = grad[j] * scale;
        m[j] = b1 * m[j] + (1.f - b1) * gs;
        v[j] = b2 * v[j] + (1.f - b2) * gs * gs;
        const float denom = sqrtf(v[j] / bc2) + eps;
        const float dm = decay_mask ? decay_mask[j] : 1.f;
        master[j] = master[j] * (1.f - lr * wd * dm) - lr * (m[j] / bc1) / denom;
        if (param_out != nullptr) {
          if (out_bf16) reinterpret_cast<__nv_bfloat16*>(param_out)[j] = __float2bfloat16(master[j]);
          else reinterpret_cast<float*>(param_out)[j] = master[j];
        }
      }
    }
  }
}

static int grid_for(long long work_items, int per_block, int max_blocks = 148 * 8) {
  long long b = (work_items + per_block - 1) / per_block;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return static_cast<int>(b);
}

// One item per thread, however many CTAs that makes.  For streams far larger than L2, whose threads have nothing to carry from item to item: CTAs that end and
// make room keep loads and stores of different items going side by side, where resident ones that walk wait for their stores' turn between their loads.
// Against 8 CTAs an SM: AdamW of 150 M elements 776 → 667 µs, the activation's backward pass (11 791 rows of 9728) 232 → 201, forward 117 → 102.
static int item_grid(long long work_items, int per_block) { return grid_for(work_items, per_block, 0x7fffffff); }

}  // namespace mb

using namespace mb;

MB_DEFINE_BOUNDS_API(mb_elementwise_bounds)

extern "C" int mb_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* res_out, float* rstd, long long T,
                              int H, float eps, cudaStream_t s) {
  if (T == 0) return 0;
  if (H % 8) return -1;
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  typedef const __nv_bfloat16* cbf;
  typedef __nv_bfloat16* bf;
  // two pieces per thread up to 4096 columns, four up to 8192 (and beyond, where the rest is read twice)
  const int pieces = H <= 4096 ? 2 : 4, threads = H <= 8192 ? (H / 8 + pieces * 32 - 1) / (pieces * 32) * 32 : 256;
  auto launch = [&](auto kern) {
    return static_cast<int>(launch_pdl(kern, dim3(static_cast<unsigned>(T)), dim3(threads), 0, s, X, (cbf)residual, (cbf)w, (bf)y, (bf)res_out, rstd, H, eps));
  };
  if (residual != nullptr) return pieces == 2 ? launch(rmsnorm_fwd_kernel<true, 2>) : launch(rmsnorm_fwd_kernel<true, 4>);
  return pieces == 2 ? launch(rmsnorm_fwd_kernel<false, 2>) : launch(rmsnorm_fwd_kernel<false, 4>);
}

// dw_partial must hold mb_rmsnorm_bwd_blocks(T) × H floats; dw_out receives the reduced weight gradient.
extern "C" int mb_rmsnorm_bwd_blocks(long long T) { return grid_for(T, 1, 148 * 4); }

static int launch_rmsnorm_bwd(const void* x, const void* w, const void* dy, const void* dres, const float* rstd, void* dx, float* dw_partial,
                              void* dw_out, int dw_fp32, long long T, int H, cudaStream_t s) {
  typedef const __nv_bfloat16* cbf;
  const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(dy) |
                         reinterpret_cast<uintptr_t>(dres) | reinterpret_cast<uintptr_t>(dx)) & 15) == 0;
  int blocks = mb_rmsnorm_bwd_blocks(T);
  // multiples of 512 up to 2560 and of 1024 up to 4096, with as many CTAs as are resident (no more than `blocks`, whose rows the buffer has)
  if (aligned && T >= 148 * 4 && H <= 4096 && (H % 1024 == 0 || (H % 512 == 0 && H <= 2560))) {
    auto launch = [&](auto kern, int per_sm) {
      blocks = 148 * per_sm;
      kern<<<blocks, 128, 0, s>>>((cbf)x, (cbf)w, (cbf)dy, (cbf)dres, rstd, reinterpret_cast<__nv_bfloat16*>(dx), dw_partial, static_cast<int>(T));
    };
    switch (H / 512) {
      case 1: launch(rmsnorm_bwd_warp_kernel<2, 1>, 3); break;
      case 2: launch(rmsnorm_bwd_warp_kernel<4, 1>, 3); break;
      case 3: launch(rmsnorm_bwd_warp_kernel<3, 2>, 3); break;
      case 4: launch(rmsnorm_bwd_warp_kernel<4, 2>, 3); break;
      case 5: launch(rmsnorm_bwd_warp_kernel<5, 2>, 2); break;
      case 6: launch(rmsnorm_bwd_warp_kernel<3, 4>, 3); break;
      default: launch(rmsnorm_bwd_warp_kernel<4, 4>, 3); break;
    }
  } else {
    rmsnorm_bwd_kernel<<<blocks, 256, 0, s>>>((cbf)x, (cbf)w, (cbf)dy, (cbf)dres, rstd, reinterpret_cast<__nv_bfloat16*>(dx), dw_partial,
                                              static_cast<int>(T), H);
  }
  colsum_kernel<<<(H + 31) / 32, 1024, 0, s>>>(dw_partial, dw_out, blocks, H, dw_fp32);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mb_rmsnorm_bwd(const void* x, const void* w, const void* dy, const void* dres, const float* rstd, void* dx,
                              float* dw_partial, void* dw_out, int dw_fp32, long long T, int H, cudaStream_t s) {
  if (T == 0) return 0;
  if (H % 8 || H > 8192) return -1;
  return launch_rmsnorm_bwd(x, w, dy, dres, rstd, dx, dw_partial, dw_out, dw_fp32, T, H, s);
}

extern "C" int mb_colsum(const float* partial, void* out, int R, int C, int out_fp32, cudaStream_t s) {
  colsum_kernel<<<(C + 31) / 32, 1024, 0, s>>>(partial, out, R, C, out_fp32);
  return static_cast<int>(cudaGetLastError());
}

// rows_ptr (optional, device): only the first min(T, *rows_ptr) rows are processed
extern "C" int mb_swiglu_fwd(const void* in, void* out, long long T, int F, const int* rows_ptr, cudaStream_t s) {
  if (T == 0) return 0;
  if (F % 8) return -1;
  return static_cast<int>(launch_pdl(swiglu_fwd_kernel, dim3(item_grid(T * (F / 8), 256)), dim3(256), 0, s,
                                     reinterpret_cast<const __nv_bfloat16*>(in), reinterpret_cast<__nv_bfloat16*>(out), T, F, rows_ptr));
}

extern "C" int mb_swiglu_bwd(const void* in, const void* dout, void* din, void* act, long long T, int F, const int* rows_ptr, cudaStream_t s) {
  if (T == 0) return 0;
  if (F % 8) return -1;
  swiglu_bwd_kernel<<<item_grid(T * (F / 8), 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(in),
                                                                reinterpret_cast<const __nv_bfloat16*>(dout),
                                                                reinterpret_cast<__nv_bfloat16*>(din), reinterpret_cast<__nv_bfloat16*>(act), T, F, rows_ptr);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mb_rope(const void* x, void* y, const int* positions, long long T, int H, int D, long long tok_stride, float theta,
                       int inverse, cudaStream_t s) {
  if (T == 0 || H == 0) return 0;
  const unsigned blocks = static_cast<unsigned>((T * H + 7) / 8);
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto Y = reinterpret_cast<__nv_bfloat16*>(y);
  if (D == 128) rope_kernel<128><<<blocks, 256, 0, s>>>(X, Y, positions, T, H, tok_stride, log2f(theta), inverse);
  else if (D == 64) rope_kernel<64><<<blocks, 256, 0, s>>>(X, Y, positions, T, H, tok_stride, log2f(theta), inverse);
  else return -1;
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mb_qk_norm_rope_fwd(const void* q, const void* k, long long q_stride, long long k_stride, const void* qw, const void* kw,
                                   const int* positions, void* qo, void* ko, float* q_rstd, float* k_rstd, long long T, int Hq, int Hk,
                                   int D, float theta, float eps, cudaStream_t s) {
  if (T == 0) return 0;
  const long long warps = T * (Hq + Hk);
  const unsigned blocks = static_cast<unsigned>((warps + 7) / 8);
  const float l2t = log2f(theta);
  if (rope_by_fours(T, Hq, Hk, Hq + Hk, D, q_stride | k_stride,
                    reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(qo) | reinterpret_cast<uintptr_t>(ko))) {
    typedef const __nv_bfloat16* cbf;
    typedef __nv_bfloat16* bf;
    return static_cast<int>(launch_pdl(qk_norm_rope_many_kernel, dim3(static_cast<unsigned>((T * ((Hq + Hk) / 4) + 7) / 8)), dim3(256), 0, s, (cbf)q, (cbf)k,
                                       (cbf)nullptr, q_stride, k_stride, 0ll, (cbf)qw, (cbf)kw, positions, (bf)qo, (bf)ko, q_rstd, k_rstd, (bf)nullptr,
                                       (bf)nullptr, (const long long*)nullptr, T, Hq, Hk, l2t, eps));
  }
  auto Q = reinterpret_cast<const __nv_bfloat16*>(q);
  auto K = reinterpret_cast<const __nv_bfloat16*>(k);
  auto QW = reinterpret_cast<const __nv_bfloat16*>(qw);
  auto KW = reinterpret_cast<const __nv_bfloat16*>(kw);
  auto QO = reinterpret_cast<__nv_bfloat16*>(qo);
  auto KO = reinterpret_cast<__nv_bfloat16*>(ko);
  if (D == 128)
    qk_norm_rope_fwd_kernel<128><<<blocks, 256, 0, s>>>(Q, K, q_stride, k_stride, QW, KW, positions, QO, KO, q_rstd, k_rstd, T, Hq, Hk, l2t, eps);
  else if (D == 64)
    qk_norm_rope_fwd_kernel<64><<<blocks, 256, 0, s>>>(Q, K, q_stride, k_stride, QW, KW, positions, QO, KO, q_rstd, k_rstd, T, Hq, Hk, l2t, eps);
  else
    return -1;
  return static_cast<int>(cudaGetLastError());
}

// Engine (no autograd) form: q/k norm + rotary, and k/v written to the paged cache [slots, Hk, D] in the same launch.
extern "C" int mb_qk_norm_rope_cache(const void* q, const void* k, const void* v, long long q_stride, long long k_stride,
                                     long long v_stride, const void* qw, const void* kw, const int* positions, void* qo, void* ko,
                                     void* kc, void* vc, const long long* slots, long long T, int Hq, int Hk, int D, float theta,
                                     float eps, cudaStream_t s) {
  if (T == 0) return 0;
  const int blocks = static_cast<int>((T * (Hq + 2 * Hk) + 7) / 8);
  const float l2t = log2f(theta);
  typedef const __nv_bfloat16* cbf;
  typedef __nv_bfloat16* bf;
  if (rope_by_fours(T, Hq, Hk, Hq + 2 * Hk, D, q_stride | k_stride | v_stride,
                    reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(qo) |
                        reinterpret_cast<uintptr_t>(ko) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)))
    return static_cast<int>(launch_pdl(qk_norm_rope_many_kernel, dim3(static_cast<unsigned>((T * ((Hq + 2 * Hk) / 4) + 7) / 8)), dim3(256), 0, s, (cbf)q,
                                       (cbf)k, (cbf)v, q_stride, k_stride, v_stride, (cbf)qw, (cbf)kw, positions, (bf)qo, (bf)ko, (float*)nullptr,
                                       (float*)nullptr, (bf)kc, (bf)vc, slots, T, Hq, Hk, l2t, eps));
  if (D == 128)
    return static_cast<int>(launch_pdl(qk_norm_rope_cache_kernel<128>, dim3(blocks), dim3(256), 0, s, (cbf)q, (cbf)k, (cbf)v, q_stride, k_stride,
                                       v_stride, (cbf)qw, (cbf)kw, positions, (bf)qo, (bf)ko, (bf)kc, (bf)vc, slots, T, Hq, Hk, l2t, eps));
  if (D == 64)
    return static_cast<int>(launch_pdl(qk_norm_rope_cache_kernel<64>, dim3(blocks), dim3(256), 0, s, (cbf)q, (cbf)k, (cbf)v, q_stride, k_stride,
                                       v_stride, (cbf)qw, (cbf)kw, positions, (bf)qo, (bf)ko, (bf)kc, (bf)vc, slots, T, Hq, Hk, l2t, eps));
  return -1;
}

extern "C" int mb_qk_norm_rope_bwd_blocks(long long T, int Hn) { return grid_for(T * Hn, 8, 148 * 4); }

// One call per tensor (q or k).  dw_partial: blocks × D floats (may be null when w is null).
extern "C" int mb_qk_norm_rope_bwd(const void* x, long long x_stride, const void* w, const float* rstd, const void* dy,
                                   const int* positions, void* dx, long long dx_stride, float* dw_partial, void* dw_out, long long T,
                                   int Hn, int D, float theta, cudaStream_t s) {
  if (T == 0) return 0;
  const int blocks = mb_qk_norm_rope_bwd_blocks(T, Hn);
  const float l2t = log2f(theta);
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto W = reinterpret_cast<const __nv_bfloat16*>(w);
  auto DY = reinterpret_cast<const __nv_bfloat16*>(dy);
  auto DX = reinterpret_cast<__nv_bfloat16*>(dx);
  if (D == 128 && w != nullptr && Hn % 4 == 0 && ((x_stride | dx_stride) & 3) == 0 &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)) & 7) == 0)
    qk_norm_rope_bwd_many_kernel<<<blocks, 256, 0, s>>>(X, x_stride, W, rstd, DY, positions, DX, dx_stride, dw_partial, T, Hn, l2t);
  else if (D == 128)
    qk_norm_rope_bwd_kernel<128><<<blocks, 256, 0, s>>>(X, x_stride, W, rstd, DY, positions, DX, dx_stride, dw_partial, T, Hn, l2t);
  else if (D == 64)
    qk_norm_rope_bwd_kernel<64><<<blocks, 256, 0, s>>>(X, x_stride, W, rstd, DY, positions, DX, dx_stride, dw_partial, T, Hn, l2t);
  else
    return -1;
  if (w != nullptr && dw_out != nullptr) colsum_kernel<<<(D + 31) / 32, 1024, 0, s>>>(dw_partial, dw_out, blocks, D, 0);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mb_kv_cache_write(const void* k, const void* v, long long k_stride, long long v_stride, void* kc, void* vc,
                                 const long long* slots, long long T, int row_elems, cudaStream_t s) {
  if (T == 0) return 0;
  if (row_elems % 8) return -1;
  kv_cache_write_kernel<<<grid_for(T * (row_elems / 8), 256), 256, 0, s>>>(
      reinterpret_cast<const __nv_bfloat16*>(k), reinterpret_cast<const __nv_bfloat16*>(v), k_stride, v_stride,
      reinterpret_cast<__nv_bfloat16*>(kc), reinterpret_cast<__nv_bfloat16*>(vc), slots, T, row_elems);
  return static_cast<int>(cudaGetLastError());
}

// See kv_gather_kernel.  kc, vc [n_slots, row_elems] bf16, slots [n]; row_elems a multiple of 8, all 16-byte aligned.
extern "C" int mb_kv_gather(const void* kc, const void* vc, const long long* slots, long long n, long long n_slots, int row_elems, void* k, void* v,
                            int* error_flag, cudaStream_t s) {
  if (n == 0) return 0;
  if (row_elems % 8) return -1;
  if ((reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15) return -2;
  return static_cast<int>(launch_pdl(kv_gather_kernel, dim3(static_cast<unsigned>((n + 31) / 32)), dim3(256), 0, s, reinterpret_cast<const __nv_bfloat16*>(kc),
                                     reinterpret_cast<const __nv_bfloat16*>(vc), slots, n, n_slots, row_elems, reinterpret_cast<__nv_bfloat16*>(k),
                                     reinterpret_cast<__nv_bfloat16*>(v), error_flag));
}

extern "C" int mb_adamw(float* master, const float* grad, float* m, float* v, const float* decay_mask, const float* scale_ptr,
                        void* param_out, int out_bf16, long long n, float lr, float b1, float b2, float eps, float wd, int step,
                        cudaStream_t s) {
  if (n == 0) return 0;
  const float bc1 = 1.f - powf(b1, static_cast<float>(step));
  const float bc2 = 1.f - powf(b2, static_cast<float>(step));
  adamw_kernel<<<item_grid(n, 1024), 256, 0, s>>>(master, grad, m, v, decay_mask, scale_ptr, param_out, out_bf16, n, lr, b1, b2, eps,
                                                wd, bc1, bc2);
  return static_cast<int>(cudaGetLastError());
}

// ---------------------------------------------------------------------------------------------
// RMSNorm backward without any allocation (declared in launch.h)
// ---------------------------------------------------------------------------------------------
// Same two kernels as mb_rmsnorm_bwd, but the per-CTA partial weight-gradient rows live in a fixed array in device
// global memory instead of a buffer supplied by the caller.  Nothing is allocated here, by CUDA or by a library.
// The array is one per device and shared by every call on that device:
//   * it keeps whatever the previous call left in it; nothing has to be cleared, because each call first writes every
//     element (rows 0..blocks-1, columns 0..H-1) that its reduction then reads;
//   * two calls that overlap in time on one device (different streams, or threads) write the same rows and race:
//     the caller orders them.
// Limit: H ≤ MB_RMSNORM_BWD_STATIC_MAX_H; larger H is refused with MB_ERR_STATIC_SCRATCH_TOO_SMALL.
static constexpr int kStaticBwdMaxBlocks = 148 * 4;   // the largest grid mb_rmsnorm_bwd_blocks() returns
static __device__ __align__(256) float g_rmsnorm_bwd_scratch[static_cast<size_t>(kStaticBwdMaxBlocks) * MB_RMSNORM_BWD_STATIC_MAX_H];

namespace {
constexpr int kMaxDevices = 64;
float* g_static_scratch_addr[kMaxDevices];   // device address of the array, looked up once per device
}  // namespace

extern "C" const char* mb_rmsnorm_bwd_static_strerror(int code) {
  switch (code) {
    case 0: return "ok";
    case -1: return "mb_rmsnorm_bwd_static: H must be a multiple of 8";
    case MB_ERR_STATIC_SCRATCH_TOO_SMALL:
      return "mb_rmsnorm_bwd_static: H exceeds MB_RMSNORM_BWD_STATIC_MAX_H (4096), the width the fixed scratch array holds; "
             "use mb_rmsnorm_bwd with a caller-provided buffer";
    case MB_ERR_STATIC_SCRATCH_SETUP: return "mb_rmsnorm_bwd_static: could not resolve the scratch array's device address";
    default: return code > 0 ? cudaGetErrorString(static_cast<cudaError_t>(code)) : "mb_rmsnorm_bwd_static: unknown error";
  }
}

extern "C" int mb_rmsnorm_bwd_static(const void* x, const void* w, const void* dy, const void* dres, const float* rstd, void* dx,
                                     void* dw_out, int dw_fp32, long long T, int H, cudaStream_t s) {
  if (H % 8) return -1;
  if (H > MB_RMSNORM_BWD_STATIC_MAX_H) return MB_ERR_STATIC_SCRATCH_TOO_SMALL;
  int dev = 0;
  cudaError_t rc = cudaGetDevice(&dev);
  if (rc != cudaSuccess) return static_cast<int>(rc);
  if (dev < 0 || dev >= kMaxDevices) return MB_ERR_STATIC_SCRATCH_SETUP;
  float* scratch = __atomic_load_n(&g_static_scratch_addr[dev], __ATOMIC_ACQUIRE);
  if (scratch == nullptr) {
    // First call on this device: resolve the symbol (this may load the module, so it belongs before any stream capture).
    void* p = nullptr;
    rc = cudaGetSymbolAddress(&p, g_rmsnorm_bwd_scratch);
    if (rc != cudaSuccess) return static_cast<int>(rc);
    if (p == nullptr) return MB_ERR_STATIC_SCRATCH_SETUP;
    scratch = static_cast<float*>(p);
    __atomic_store_n(&g_static_scratch_addr[dev], scratch, __ATOMIC_RELEASE);   // racing first calls store the same value
  }
  if (T == 0) return 0;
  if (mb_rmsnorm_bwd_blocks(T) > kStaticBwdMaxBlocks) return MB_ERR_STATIC_SCRATCH_TOO_SMALL;
  return launch_rmsnorm_bwd(x, w, dy, dres, rstd, dx, scratch, dw_out, dw_fp32, T, H, s);
}
