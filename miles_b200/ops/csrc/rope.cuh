// Per-head RMSNorm and rotation of one row by one warp.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace mb {

// (x1, x2) turned by the angle of cosine c and sine s.  The contraction is spelled out: left to the compiler, two kernels round the same token in
// two ways.
__device__ __forceinline__ float2 rotate_pair(float x1, float x2, float c, float s) {
  return make_float2(__fmaf_rn(x1, c, -__fmul_rn(x2, s)), __fmaf_rn(x1, s, __fmul_rn(x2, c)));
}

// Lane's D / 64 columns of each half of rmsnorm(src) · w (w null: src), rotated by the position's angles.
template <int D>
__device__ __forceinline__ void norm_rope_values(const __nv_bfloat16* __restrict__ src, const __nv_bfloat16* __restrict__ w, float pos, float log2_theta,
                                                 float eps, float* rstd_out, int lane, __nv_bfloat16 (&o1)[D / 64], __nv_bfloat16 (&o2)[D / 64]) {
  constexpr int EPL = D / 64;
  float a[EPL], b[EPL];
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < EPL; ++e) {
    a[e] = __bfloat162float(src[lane * EPL + e]);
    b[e] = __bfloat162float(src[D / 2 + lane * EPL + e]);
    ss += a[e] * a[e] + b[e] * b[e];
  }
  float rstd = 1.f;
  if (w != nullptr) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    rstd = rsqrtf(ss / D + eps);
    if (rstd_out != nullptr && lane == 0) *rstd_out = rstd;
  }
#pragma unroll
  for (int e = 0; e < EPL; ++e) {
    const int j = lane * EPL + e;
    float x1 = a[e], x2 = b[e];
    if (w != nullptr) {
      x1 = __bfloat162float(__float2bfloat16(x1 * rstd * __bfloat162float(w[j])));
      x2 = __bfloat162float(__float2bfloat16(x2 * rstd * __bfloat162float(w[D / 2 + j])));
    }
    const float inv_freq = exp2f(-log2_theta * (2.f * j) / D);
    float s, c;
    sincosf(pos * inv_freq, &s, &c);
    const float2 r = rotate_pair(x1, x2, c, s);
    o1[e] = __float2bfloat16(r.x);
    o2[e] = __float2bfloat16(r.y);
  }
}

}  // namespace mb
