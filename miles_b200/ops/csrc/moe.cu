// MoE routing and token permutation around the grouped tcgen05 GEMMs.
//   router_topk   softmax over all experts + top-k (+ renormalisation); one warp per token
//   norm_router   add + RMSNorm + router logits + top-k of a decode step, one CTA per token
//   moe_align     counting sort of (token, slot) pairs by expert into 128-row-padded segments; no host sync:
//                 buffers are sized for the worst case and the tile → expert table tells the GEMM what to skip
//   moe_gather    x_perm[row] = x[token(row)]            (pad rows zero-filled)
//   moe_combine   out[t] = Σ_j w[t,j] · y_perm[row(t,j)]   (gather form: deterministic, no atomics)
//   moe_glu_bwd   the experts' activation in the backward pass, with the gradient of the gate weights
//   moe_combine_bwd  dy_perm[row] = w · dout[token(row)],  dw[t,j] = ⟨dout[t], y_perm[row(t,j)]⟩
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.h"
#include "debug.cuh"
#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {

typedef __nv_bfloat16 bf16;
static constexpr int kPad = 128;

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float wmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------------------------------------
// The k most probable experts of one token by one warp: lane holds experts lane, lane + 32, … of the logits v (−inf beyond E).  On return lane j < K
// has choice j (−1: a row of NaNs has no winner) and its weight.  `recorded`: lane j's recorded choice or a negative number; recorded choices replace
// the top-k and their weights come from these logits; a token without any is chosen afresh.  A choice outside [0, E) of another token is no record of
// this model: it raises the error flag (72), and expert 0 with weight 0 stands in its place, so that nothing behind reads out of range.
template <int EPL>  // experts per lane = E / 32
__device__ __forceinline__ void softmax_topk(float (&v)[EPL], int E, int K, int normalize, int recorded, float* probs, int* error_flag, int& choice,
                                             float& weight) {
  const int lane = threadIdx.x & 31;
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < EPL; ++i) mx = fmaxf(mx, v[i]);
  mx = wmax(mx);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    v[i] = (i * 32 + lane < E) ? __expf(v[i] - mx) : 0.f;
    s += v[i];
  }
  s = wsum(s);
  const float inv = 1.f / s;
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    v[i] *= inv;
    if (probs != nullptr && i * 32 + lane < E) probs[i * 32 + lane] = v[i];
  }
  float wsel = 0.f, mine_w = 0.f;
  int mine_i = 0;
  const bool replayed = __any_sync(0xffffffffu, recorded >= 0);
  for (int j = 0; replayed && j < K; ++j) {
    const int e = __shfl_sync(0xffffffffu, recorded, j);
    float p = 0.f;
#pragma unroll
    for (int i = 0; i < EPL; ++i) p = (e >> 5) == i ? v[i] : p;
    p = __shfl_sync(0xffffffffu, p, e & 31);
    const bool valid = e >= 0 && e < E;
    if (!valid) p = 0.f;
    wsel += p;
    if (lane == j) { mine_w = p; mine_i = valid ? e : 0; }
    if (!valid && lane == 0) atomicCAS(error_flag, 0, 72);
  }
  for (int j = 0; !replayed && j < K; ++j) {
    float bv = -1.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const int e = i * 32 + lane;
      if (e < E && (v[i] > bv)) { bv = v[i]; bi = e; }   // ascending e → ties keep the lower id
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    // remove the winner (unrolled compare keeps v[] in registers)
#pragma unroll
    for (int i = 0; i < EPL; ++i)
      if (i * 32 + lane == bi) v[i] = -2.f;
    if (bi == 0x7fffffff) { bv = 0.f; bi = -1; }   // a row of NaNs has no winner: slot left empty (−1), never an id out of range
    wsel += bv;
    if (lane == j) { mine_w = bv; mine_i = bi; }
  }
  choice = mine_i;
  weight = normalize ? mine_w / fmaxf(wsel, 1e-20f) : mine_w;
}

// `replay`: recorded choices, rows `replay_row` apart.  In one launch where softmax, gather, sum and division were kernels of their own behind a host
// synchronisation that asked whether any row was without: 12 launches and a round trip per layer.
template <int EPL>
__global__ void __launch_bounds__(256) router_topk_kernel(const float* logits, float* probs,
                                                          float* topk_w, int* topk_idx, long long T, int E,
                                                          int K, int normalize, const int* replay, long long replay_row,
                                                          int* error_flag) {
  pdl_trigger();
  pdl_wait();
  const long long t = (blockIdx.x * 256ll + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  float v[EPL];
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    const int e = i * 32 + lane;
    v[i] = (e < E) ? logits[t * E + e] : -INFINITY;
  }
  int choice;
  float weight;
  softmax_topk<EPL>(v, E, K, normalize, replay != nullptr && lane < K ? replay[t * replay_row + lane] : -1, probs != nullptr ? probs + t * E : nullptr,
                    error_flag, choice, weight);
  if (lane < K) {
    topk_idx[t * K + lane] = choice;
    topk_w[t * K + lane] = weight;
  }
}

// A decode step's way from a sublayer's output to its experts in one launch, a CTA per token: h = bf16(x + residual) → sum, bf16(h / rms · norm_w) →
// normed, router logits (h · norm_w) · W / rms with fp32 operands throughout, softmax, top-k.  What bounds it is the chain of latencies (row, sum of
// squares, router rows, top-k), so each is paid once: a warp has one expert, whose row it requests before the dependency wait (weights).
// Norm, logits and top-k as launches of their own took 7.1 µs of a decode step's layer of 1 row (16 experts, hidden 2048), 10.0 of 7 and 9.2 of 61;
// this one 4.4 to 4.6.
static constexpr int kRouterWarps = 16, kRouterMaxH = 4096;

__global__ void __launch_bounds__(kRouterWarps * 32) norm_router_kernel(const bf16* x, const bf16* residual, const bf16* norm_w,
                                                                        const bf16* W, float eps, int H, int E, int K, int normalize, int static_w,
                                                                        bf16* sum, bf16* normed, float* topk_w, int* topk_idx) {
  constexpr int kPieces = kRouterMaxH / 256;              // 16-byte pieces of a router row per lane
  __shared__ __align__(16) float hs[kRouterMaxH];         // h · norm_w
  __shared__ float part[kRouterWarps], logit[32];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long t = blockIdx.x;
  uint4 w[kPieces];
  if (!static_w) pdl_wait();
#pragma unroll
  for (int i = 0; i < kPieces; ++i)
    if (warp < E && i * 256 + lane * 8 < H) w[i] = *reinterpret_cast<const uint4*>(W + static_cast<long long>(warp) * H + i * 256 + lane * 8);
  const int at = threadIdx.x * 8;                         // H ≤ 4096: one piece of the row per thread
  auto two = [](uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); };
  uint4 nw = make_uint4(0, 0, 0, 0);
  if (at < H) nw = *reinterpret_cast<const uint4*>(norm_w + at);
  if (static_w) pdl_wait();
  uint4 h = make_uint4(0, 0, 0, 0);
  uint32_t* hp = &h.x;
  const uint32_t* np = &nw.x;
  float ss = 0.f;
  if (at < H) {
    h = *reinterpret_cast<const uint4*>(x + t * H + at);
    if (residual != nullptr) {
      const uint4 r = *reinterpret_cast<const uint4*>(residual + t * H + at);
      const uint32_t* rp = &r.x;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = two(hp[i]), b = two(rp[i]);
        hp[i] = pack_bf16x2(a.x + b.x, a.y + b.y);
      }
      *reinterpret_cast<uint4*>(sum + t * H + at) = h;
    }
    float f[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = two(hp[i]), b = two(np[i]);
      ss += a.x * a.x + a.y * a.y;
      f[2 * i] = a.x * b.x;
      f[2 * i + 1] = a.y * b.y;
    }
    *reinterpret_cast<float4*>(hs + at) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(hs + at + 4) = make_float4(f[4], f[5], f[6], f[7]);
  }
  ss = wsum(ss);
  if (lane == 0) part[warp] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < kRouterWarps; ++i) ss += part[i];
  const float rstd = rsqrtf(ss / H + eps);
  if (warp < E) {
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
      if (i * 256 + lane * 8 >= H) continue;
      const float4 a = *reinterpret_cast<const float4*>(hs + i * 256 + lane * 8), b = *reinterpret_cast<const float4*>(hs + i * 256 + lane * 8 + 4);
      const float2 w0 = two(w[i].x), w1 = two(w[i].y), w2 = two(w[i].z), w3 = two(w[i].w);
      acc += (a.x * w0.x + a.y * w0.y) + (a.z * w1.x + a.w * w1.y) + ((b.x * w2.x + b.y * w2.y) + (b.z * w3.x + b.w * w3.y));
    }
    acc = wsum(acc);
    if (lane == 0) logit[warp] = acc * rstd;
  }
  if (at < H) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = two(hp[i]), b = two(np[i]);
      o[i] = pack_bf16x2(a.x * rstd * b.x, a.y * rstd * b.y);
    }
    *reinterpret_cast<uint4*>(normed + t * H + at) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  __syncthreads();
  if (warp != 0) return;
  float v[1] = {lane < E ? logit[lane] : -INFINITY};
  int choice;
  float weight;
  softmax_topk<1>(v, E, K, normalize, -1, nullptr, nullptr, choice, weight);
  if (lane < K) {
    topk_idx[t * K + lane] = choice;
    topk_w[t * K + lane] = weight;
  }
}

// ---------------------------------------------------------------------------------------------
// Single-CTA counting sort.  idx[n] holds global expert ids; local expert = id − expert_offset, others skipped.
// Outputs: seg_offsets[E+1] (segments padded to `pad` rows), tile_expert[max_rows / pad], row_src[max_rows], dst_row[n].
__global__ void __launch_bounds__(1024) moe_align_kernel(const int* idx, int n, const int* n_ptr, int E,
                                                         int expert_offset, int* seg_offsets, int* tile_expert,
                                                         int* row_src, int* dst_row, int max_rows, int pad) {
  extern __shared__ int sh[];  // counts[E], cursor[E], seg[E+1]
  pdl_trigger();
  pdl_wait();
  if (n_ptr != nullptr) n = min(n, *n_ptr);   // device-side entry count (expert-parallel receive buffers)
  int* counts = sh;
  int* cursor = sh + E;
  int* seg = sh + 2 * E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) { counts[e] = 0; cursor[e] = 0; }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int e = idx[i] - expert_offset;
    if (e >= 0 && e < E) atomicAdd(&counts[e], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int off = 0;
    for (int e = 0; e < E; ++e) {
      seg[e] = off;
      off += (counts[e] + pad - 1) / pad * pad;
    }
    seg[E] = off;
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) seg_offsets[e] = seg[e];
  const int max_tiles = max_rows / pad;
  for (int t = threadIdx.x; t < max_tiles; t += blockDim.x) {
    const int row = t * pad;
    int ex = -1;
    if (row < seg[E]) {
      int lo = 0, hi = E;   // last e with seg[e] <= row
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (seg[mid] <= row) lo = mid; else hi = mid;
      }
      ex = lo;
    }
    tile_expert[t] = ex;
  }
  // rows at or beyond seg[E] are never read (every consumer stops at seg[E]), so only the used prefix is cleared
  for (int r = threadIdx.x; r < seg[E] && r < max_rows; r += blockDim.x) row_src[r] = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int e = idx[i] - expert_offset;
    int row = -1;
    if (e >= 0 && e < E) {
      row = seg[e] + atomicAdd(&cursor[e], 1);
      row_src[row] = i;
    }
    dst_row[i] = row;
  }
}

// The same sort by a cluster of CTAs (8 of 32 warps, or one of 8 to 32), for E ≤ kMaxSortExperts.  Every warp owns a contiguous range of the pairs and
// counts it into its own histogram (lanes with the same expert are found with match.any: no atomics); after the counts have been added up
// across warps and, through distributed shared memory, across CTAs, it walks its range again and hands out rows.  Pairs keep their order
// within an expert, so the result does not depend on timing.  One CTA with shared-memory atomics on 16 counters was bound by their
// serialisation: 58 064 pairs, 16 experts: 44 → 17.5 µs (fewer: `mb_moe_align_pad`).
static constexpr int kMaxSortExperts = 256, kSortWarps = 32;

__global__ void __launch_bounds__(kSortWarps * 32) moe_sort_kernel(const int* idx, int n, const int* n_ptr, int E, int expert_offset, int* seg_offsets,
                                                                   int* tile_expert, int* row_src, int* dst_row, int max_rows, int pad, int ctas) {
  extern __shared__ int sh[];
  pdl_trigger();
  pdl_wait();
  if (n_ptr != nullptr) n = min(n, *n_ptr);
  int* cursor = sh;                         // [warp][E]: counts, then the next row
  const int nw = static_cast<int>(blockDim.x) >> 5;
  int* mine = cursor + nw * E;              // [E] this CTA's counts (read by the other CTAs)
  int* all = mine + E;                      // [E] everybody's
  int* seg = all + E;                       // [E + 1]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = static_cast<int>(blockIdx.x);
  int* my = cursor + warp * E;
  for (int e = lane; e < E; e += 32) my[e] = 0;
  __syncwarp();
  const int warps = ctas * nw, per = ((n + warps - 1) / warps + 31) / 32 * 32;
  const int begin = min(n, (rank * nw + warp) * per), end = min(n, begin + per);
  auto expert_at = [&](int i) {
    const int e = i < end ? idx[i] - expert_offset : -1;
    return e >= 0 && e < E ? e : -1;
  };
  int e4[4], at[4];                         // a warp's only (or last) four rounds: expert, place among the warp's pairs of that expert
  for (int i0 = begin; i0 < end; i0 += 128) {
#pragma unroll
    for (int u = 0; u < 4; ++u) e4[u] = expert_at(i0 + u * 32 + lane);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t same = __match_any_sync(0xffffffffu, e4[u]);
      if (e4[u] >= 0) at[u] = my[e4[u]] + __popc(same & ((1u << lane) - 1));
      __syncwarp();
      if (e4[u] >= 0 && __ffs(same) - 1 == lane) my[e4[u]] += __popc(same);
      __syncwarp();
    }
  }
  __syncthreads();
  // counts of the warps before, per expert (eight at a time: the loads go out together; the number of warps is a multiple of eight)
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int sum = 0;
    for (int w0 = 0; w0 < nw; w0 += 8) {
      int c[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) c[w] = cursor[(w0 + w) * E + e];
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        cursor[(w0 + w) * E + e] = sum;
        sum += c[w];
      }
    }
    mine[e] = sum;
  }
  __syncthreads();
  if (ctas > 1) cluster_sync();
  // … and of the CTAs before
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int sum = 0, before = 0;
    for (int c = 0; c < ctas; ++c) {
      int v = mine[e];
      if (ctas > 1) asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(smem_of_rank(mine + e, c)));
      if (c < rank) before += v;
      sum += v;
    }
    all[e] = sum;
    if (before != 0)
      for (int w = 0; w < nw; ++w) cursor[w * E + e] += before;
  }
  __syncthreads();
  if (ctas > 1) cluster_sync();             // the last read of another CTA's memory
  if (warp == 0) {
    int off = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane, rows = e < E ? (all[e] + pad - 1) / pad * pad : 0;
      int sum = rows;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += x;
      }
      if (e < E) seg[e] = off + sum - rows;
      off += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) seg[E] = off;
  }
  __syncthreads();
  const int thread = rank * blockDim.x + threadIdx.x, threads = ctas * blockDim.x;
  for (int e = thread; e <= E; e += threads) seg_offsets[e] = seg[e];
  for (int t = thread; t < max_rows / pad; t += threads) {
    const int row = t * pad;
    int ex = -1;
    if (row < seg[E]) {
      int lo = 0, hi = E;   // last e with seg[e] <= row
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (seg[mid] <= row) lo = mid; else hi = mid;
      }
      ex = lo;
    }
    tile_expert[t] = ex;
  }
  // the rows behind a segment's last pair (rows at or beyond seg[E] are never read)
  for (int e = rank * nw + warp; e < E; e += warps)
    for (int r = seg[e] + all[e] + lane; r < seg[e + 1] && r < max_rows; r += 32) row_src[r] = -1;
  if (per <= 128) {
    if (begin < end) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = begin + u * 32 + lane, row = e4[u] >= 0 ? seg[e4[u]] + my[e4[u]] + at[u] : -1;
        if (row >= 0) row_src[row] = i;
        if (i < end) dst_row[i] = row;
      }
    }
    return;
  }
  for (int i0 = begin; i0 < end; i0 += 128) {
    int e[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) e[u] = expert_at(i0 + u * 32 + lane);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * 32 + lane;
      const uint32_t same = __match_any_sync(0xffffffffu, e[u]);
      int row = -1;
      if (e[u] >= 0) {
        row = seg[e[u]] + my[e[u]] + __popc(same & ((1u << lane) - 1));
        row_src[row] = i;
      }
      __syncwarp();
      if (e[u] >= 0 && __ffs(same) - 1 == lane) my[e[u]] += __popc(same);
      __syncwarp();
      if (i < end) dst_row[i] = row;
    }
  }
}

// A warp moves kVec 16-byte pieces per lane of a row at a time, all of them in flight together: a CTA per row with one piece per thread waits
// for its index, its row and its store one after another (half of the bandwidth).
static constexpr int kVec = 8;

// x_perm[row, :] = x[row_src[row] / k, :]  (zero for pad rows inside used segments; rows ≥ total untouched)
// 58 064 rows of 2048: 80 → 53 µs.
__global__ void __launch_bounds__(256) moe_gather_kernel(const bf16* x, bf16* x_perm, const int* row_src, const int* seg_offsets, int E, int k, int H,
                                                         int max_rows) {
  pdl_trigger();
  pdl_wait();
  const int total = min(seg_offsets[E], max_rows), nvec = H / 8, lane = threadIdx.x & 31;
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < total; row += gridDim.x * 8) {
    const int src = row_src[row];
    const bool real = src >= 0 && dbg::in_bounds(dbg::kMoePairs, src, 201);
    uint4* dst = reinterpret_cast<uint4*>(x_perm + static_cast<long long>(row) * H);
    const uint4* s = reinterpret_cast<const uint4*>(x + static_cast<long long>(real ? src / k : 0) * H);
    for (int v0 = lane; v0 < nvec; v0 += 32 * kVec) {
      uint4 r[kVec];
#pragma unroll
      for (int u = 0; u < kVec; ++u) r[u] = real && v0 + u * 32 < nvec ? s[v0 + u * 32] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < kVec; ++u)
        if (v0 + u * 32 < nvec) dst[v0 + u * 32] = r[u];
    }
  }
}

// out[t, :] = Σ_j w[t,j] · y_perm[dst_row[t·k+j], :]   (w == nullptr → weights 1)
// identity_rows: dst_row only says whether pair p took part (≥ 0); its row is p itself (per-pair return buffers).
// Eight choices at a time: their rows are requested together and added in order: 7258 tokens × 8 × 2048: 67 → 57 µs
// (61 tokens: 5.0 → 3.0).
__global__ void __launch_bounds__(256) moe_combine_kernel(const bf16* y_perm, const float* w, const int* dst_row, bf16* out, long long T, int k, int H,
                                                          int identity_rows) {
  pdl_trigger();
  pdl_wait();
  const int nvec = H / 8;
  for (long long t = blockIdx.x; t < T; t += gridDim.x) {
    for (int v = threadIdx.x; v < nvec; v += 256) {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int j0 = 0; j0 < k; j0 += 8) {
        uint4 raw[8];
        float wj[8];
        bool in[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const long long at = t * k + j0 + u;
          int row = j0 + u < k ? dst_row[at] : -1;
          in[u] = row >= 0;
          if (identity_rows) row = static_cast<int>(at);
          wj[u] = in[u] && w != nullptr ? w[at] : 1.f;
          raw[u] = in[u] ? *reinterpret_cast<const uint4*>(y_perm + static_cast<long long>(row) * H + v * 8) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (!in[u]) continue;
          const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(p[i]);
            acc[2 * i] += wj[u] * f.x;
            acc[2 * i + 1] += wj[u] * f.y;
          }
        }
      }
      uint4 o;
      __nv_bfloat162* q = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      *reinterpret_cast<uint4*>(out + t * H + v * 8) = o;
    }
  }
}

// The same with the residual stream's add and the next RMSNorm behind it: the weighted sum never goes to memory.  A CTA per token, whose threads own the
// columns that rmsnorm_fwd_kernel's own (two pieces each, H ≤ 4096): sums and roundings are those of the two kernels it stands for.  What bounds it: the rows
// of y.  7258 tokens × 8 × 2048: 49 + 19 → 56 µs, 17 829: 112 + 45 → 129 (123 at the memory's speed; a warp per token 61 and 130).
__global__ void __launch_bounds__(256) moe_combine_norm_kernel(const bf16* y_perm, const float* w, const int* dst_row, const bf16* residual,
                                                               const bf16* __restrict__ norm_w, bf16* y, bf16* res_out, int k, int H, float eps) {
  constexpr int N = 2;
  __shared__ float sh[8];
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, nvec = H / 8, nt = blockDim.x;
  const long long t = blockIdx.x;
  uint4 v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int c = threadIdx.x + nt * i;
    if (c < nvec) v[i] = reinterpret_cast<const uint4*>(residual + t * H)[c];
  }
  const int row0 = lane < k ? dst_row[t * k + lane] : -1;              // the first 32 choices; more are read where they are used
  const float w0 = lane < k ? w[t * k + lane] : 0.f;
  float acc[N][8] = {};
  for (int j0 = 0; j0 < k; j0 += 8) {
    uint4 raw[8][N];
    float wj[8];
    bool in[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u;
      int row = __shfl_sync(0xffffffffu, row0, j & 31);
      wj[u] = __shfl_sync(0xffffffffu, w0, j & 31);
      if (j >= 32 && j < k) { row = dst_row[t * k + j]; wj[u] = w[t * k + j]; }
      in[u] = j < k && row >= 0;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int c = threadIdx.x + nt * i;
        raw[u][i] = in[u] && c < nvec ? reinterpret_cast<const uint4*>(y_perm + static_cast<long long>(row) * H)[c] : make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (in[u])
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&raw[u][i])[e]);
            acc[i][2 * e] += wj[u] * f.x;
            acc[i][2 * e + 1] += wj[u] * f.y;
          }
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int c = threadIdx.x + nt * i;
    if (c < nvec) {
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v[i]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 a = __bfloat1622float2(__floats2bfloat162_rn(acc[i][2 * e], acc[i][2 * e + 1])), b = __bfloat1622float2(h[e]);
        h[e] = __floats2bfloat162_rn(a.x + b.x, a.y + b.y);
        const float2 f = __bfloat1622float2(h[e]);
        ss += f.x * f.x + f.y * f.y;
      }
      reinterpret_cast<uint4*>(res_out + t * H)[c] = v[i];
    }
  }
  ss = wsum(ss);
  if (lane == 0) sh[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i < nt / 32) ss += sh[i];
  const float rstd = rsqrtf(ss / H + eps);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int c = threadIdx.x + nt * i;
    if (c >= nvec) continue;
    const uint4 wv = reinterpret_cast<const uint4*>(norm_w)[c];
    uint4 o;
    __nv_bfloat162* q = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&v[i])[e]), b = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&wv)[e]);
      q[e] = __floats2bfloat162_rn(a.x * rstd * b.x, a.y * rstd * b.y);
    }
    reinterpret_cast<uint4*>(y + t * H)[c] = o;
  }
}

// dy_perm[row] = w[flat]·dout[token];  dw[flat] = ⟨dout[token], y_perm[row]⟩   (one warp per permuted row)
__global__ void __launch_bounds__(256) moe_combine_bwd_kernel(const bf16* dout, const bf16* y_perm, const float* w, const int* row_src,
                                                              const int* seg_offsets, int E, bf16* dy_perm, float* dw, int k, int H, int max_rows) {
  const int total = min(seg_offsets[E], max_rows), nvec = H / 8, lane = threadIdx.x & 31;
  constexpr int kHalf = kVec / 2;
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < total; row += gridDim.x * 8) {
    const int flat = row_src[row];
    const bool real = flat >= 0;
    uint4* dst = reinterpret_cast<uint4*>(dy_perm + static_cast<long long>(row) * H);
    const uint4* g = reinterpret_cast<const uint4*>(dout + static_cast<long long>(real ? flat / k : 0) * H);
    const uint4* y = reinterpret_cast<const uint4*>(y_perm + static_cast<long long>(row) * H);
    const float wj = real ? w[flat] : 0.f;
    float dot = 0.f;
    for (int v0 = lane; v0 < nvec; v0 += 32 * kHalf) {
      uint4 gr[kHalf], yr[kHalf];
#pragma unroll
      for (int u = 0; u < kHalf; ++u) {
        const bool in = real && v0 + u * 32 < nvec;
        gr[u] = in ? g[v0 + u * 32] : make_uint4(0, 0, 0, 0);
        yr[u] = in && dw != nullptr ? y[v0 + u * 32] : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < kHalf; ++u) {
        if (v0 + u * 32 >= nvec) continue;
        const __nv_bfloat162* gp = reinterpret_cast<const __nv_bfloat162*>(&gr[u]);
        const __nv_bfloat162* yp = reinterpret_cast<const __nv_bfloat162*>(&yr[u]);
        uint4 o = make_uint4(0, 0, 0, 0);
        __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(&o);
        if (real) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 gf = __bfloat1622float2(gp[i]), yf = __bfloat1622float2(yp[i]);
            dot += gf.x * yf.x + gf.y * yf.y;
            op[i] = __floats2bfloat162_rn(gf.x * wj, gf.y * wj);
          }
        }
        dst[v0 + u * 32] = o;
      }
    }
    if (dw != nullptr && real) {
      dot = wsum(dot);
      if (lane == 0) dw[flat] = dot;
    }
  }
}

// The experts' activation in the backward pass, one warp per permuted row of a pair with weight w: a = silu(gate) · up from h1 = [gate, up],
// d = the row of dout · W2 (in act_w's place):  dw[flat] = ⟨d, a⟩,  dh1 = gradient of h1 for w · d,  act_w = w · a (what W2's gradient multiplies dout
// with).  Pad rows give zeros.  What bounds it: six passes of the row's width over memory.  It stands for the activation's recomputation, its
// backward and the sums ⟨dout, y⟩ over rows of y, which nobody has to keep any more: 96 600 rows of 768, hidden 2048: 90 + 156 + 170 µs → 164
// and 110 for the gather of the rows of dout.
__global__ void __launch_bounds__(256) moe_glu_bwd_kernel(const bf16* h1, bf16* act_w, bf16* dh1, const float* w, const int* row_src, const int* seg_offsets, int E,
                                                          float* dw, int F, int max_rows) {
  constexpr int U = 3;
  const int total = min(seg_offsets[E], max_rows), nvec = F / 8, lane = threadIdx.x & 31;
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < total; row += gridDim.x * 8) {
    const int flat = row_src[row];
    const bool real = flat >= 0;
    const float wj = real ? w[flat] : 0.f;
    const uint4* gate = reinterpret_cast<const uint4*>(h1 + 2ll * row * F);
    uint4* d = reinterpret_cast<uint4*>(act_w + static_cast<long long>(row) * F);
    uint4* out = reinterpret_cast<uint4*>(dh1 + 2ll * row * F);
    float dot = 0.f;
    for (int v0 = lane; v0 < nvec; v0 += 32 * U) {
      uint4 gr[U], ur[U], dr[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool in = real && v0 + u * 32 < nvec;
        gr[u] = in ? gate[v0 + u * 32] : make_uint4(0, 0, 0, 0);
        ur[u] = in ? gate[nvec + v0 + u * 32] : make_uint4(0, 0, 0, 0);
        dr[u] = in ? d[v0 + u * 32] : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (v0 + u * 32 >= nvec) continue;
        const __nv_bfloat162 *gp = reinterpret_cast<const __nv_bfloat162*>(&gr[u]), *up = reinterpret_cast<const __nv_bfloat162*>(&ur[u]),
                             *dp = reinterpret_cast<const __nv_bfloat162*>(&dr[u]);
        uint4 ao, go, uo;
        __nv_bfloat162 *ap = reinterpret_cast<__nv_bfloat162*>(&ao), *gq = reinterpret_cast<__nv_bfloat162*>(&go), *uq = reinterpret_cast<__nv_bfloat162*>(&uo);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 g = __bfloat1622float2(gp[i]), x = __bfloat1622float2(up[i]), e = __bfloat1622float2(dp[i]);
          const float s0 = 1.f / (1.f + __expf(-g.x)), s1 = 1.f / (1.f + __expf(-g.y));
          const float a0 = g.x * s0 * x.x, a1 = g.y * s1 * x.y;
          const float2 a = __bfloat1622float2(__floats2bfloat162_rn(a0, a1));            // as the forward product read it
          dot += e.x * a.x + e.y * a.y;
          ap[i] = __floats2bfloat162_rn(wj * a0, wj * a1);
          gq[i] = __floats2bfloat162_rn(wj * e.x * x.x * s0 * (1.f + g.x * (1.f - s0)), wj * e.y * x.y * s1 * (1.f + g.y * (1.f - s1)));
          uq[i] = __floats2bfloat162_rn(wj * e.x * g.x * s0, wj * e.y * g.y * s1);
        }
        d[v0 + u * 32] = ao;
        out[v0 + u * 32] = go;
        out[nvec + v0 + u * 32] = uo;
      }
    }
    if (real) {
      dot = wsum(dot);
      if (lane == 0) dw[flat] = dot;
    }
  }
}

}  // namespace mb

using namespace mb;

MB_DEFINE_BOUNDS_API(mb_moe_bounds)

extern "C" int mb_router_topk(const float* logits, float* probs, float* topk_w, int* topk_idx, long long T, int E, int K,
                              int normalize, const int* replay, long long replay_row, int* error_flag, cudaStream_t s) {
  if (T == 0) return 0;
  if (E > 256 || K > 32) return -1;
  const unsigned blocks = static_cast<unsigned>((T + 7) / 8);
  const int epl = (E + 31) / 32;
  cudaError_t e;
  if (epl <= 1) e = launch_pdl(router_topk_kernel<1>, dim3(blocks), dim3(256), 0, s, logits, probs, topk_w, topk_idx, T, E, K, normalize, replay, replay_row, error_flag);
  else if (epl <= 2) e = launch_pdl(router_topk_kernel<2>, dim3(blocks), dim3(256), 0, s, logits, probs, topk_w, topk_idx, T, E, K, normalize, replay, replay_row, error_flag);
  else if (epl <= 4) e = launch_pdl(router_topk_kernel<4>, dim3(blocks), dim3(256), 0, s, logits, probs, topk_w, topk_idx, T, E, K, normalize, replay, replay_row, error_flag);
  else e = launch_pdl(router_topk_kernel<8>, dim3(blocks), dim3(256), 0, s, logits, probs, topk_w, topk_idx, T, E, K, normalize, replay, replay_row, error_flag);
  return static_cast<int>(e);
}

// See norm_router_kernel.  x, residual (or null), sum (null without a residual), normed [T, H] bf16, norm_w [H], W [E, H] bf16, all 16-byte aligned;
// H ≤ 4096 and a multiple of 8, K ≤ E ≤ 16.  static_w: no kernel that may still run on the stream writes W or norm_w.
extern "C" int mb_norm_router(const void* x, const void* residual, const void* norm_w, const void* W, float eps, int T, int H, int E, int K, int normalize,
                              int static_w, void* sum, void* normed, float* topk_w, int* topk_idx, cudaStream_t s) {
  if (T <= 0) return 0;
  if (E < 1 || E > kRouterWarps || K < 1 || K > E || H < 8 || H > kRouterMaxH || H % 8 || (residual != nullptr && sum == nullptr)) return -1;
  const uintptr_t pointers = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(norm_w) |
                             reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(sum) | reinterpret_cast<uintptr_t>(normed);
  if (pointers & 15) return -2;
  return static_cast<int>(launch_pdl(norm_router_kernel, dim3(T), dim3(kRouterWarps * 32), 0, s, reinterpret_cast<const bf16*>(x), reinterpret_cast<const bf16*>(residual),
                                     reinterpret_cast<const bf16*>(norm_w), reinterpret_cast<const bf16*>(W), eps, H, E, K, normalize, static_w,
                                     reinterpret_cast<bf16*>(sum), reinterpret_cast<bf16*>(normed), topk_w, topk_idx));
}

// pad: rows every expert segment is rounded up to (128 for the training GEMMs, 16/32/64 for the decode-sized grouped GEMM)
extern "C" int mb_moe_align_pad(const int* idx, int n, const int* n_ptr, int E, int expert_offset, int* seg_offsets, int* tile_expert,
                                int* row_src, int* dst_row, int max_rows, int pad, int ordered, cudaStream_t s) {
  if (E > 2048 || pad <= 0) return -1;
  // Where the order of a segment's rows does not matter (nothing is summed over them), the counters are faster as long as they are few, one
  // thread adds up the segments, and the pairs are (488 pairs: 8 experts 2.5 against 3.4 µs, 16 3.0 / 3.8, 32 4.0 / 4.3, but 64 6.0 / 5.6;
  // 16 experts: 2048 pairs 3.9 / 5.4, 4096 4.9 / 7.1, 8192 7.1 / 6.4)
  if (E <= kMaxSortExperts && (ordered || E > 32 || n > 4096)) {
    // eight CTAs from where one's passes over its range outlast two cluster barriers; the warps' histograms take 128 bytes per expert
    // and a warp is worth its row of the histogram from two passes over 32 pairs
    const int ctas = n > 4096 ? 8 : 1, warps = n > 1024 ? kSortWarps : n > 512 ? 16 : 8;
    const size_t bytes = (warps * E + 3 * E + 1) * sizeof(int);
    static const cudaError_t configured = cudaFuncSetAttribute(moe_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                               static_cast<int>((kSortWarps + 3) * kMaxSortExperts * sizeof(int) + 16));
    if (configured != cudaSuccess) return static_cast<int>(configured);
    return static_cast<int>(launch_pdl_cluster(moe_sort_kernel, dim3(ctas), dim3(warps * 32), ctas, bytes, s, idx, n, n_ptr, E, expert_offset,
                                               seg_offsets, tile_expert, row_src, dst_row, max_rows, pad, ctas));
  }
  return static_cast<int>(launch_pdl(moe_align_kernel, dim3(1), dim3(1024), (3 * E + 1) * sizeof(int), s, idx, n, n_ptr, E, expert_offset,
                                     seg_offsets, tile_expert, row_src, dst_row, max_rows, pad));
}

extern "C" int mb_moe_align(const int* idx, int n, const int* n_ptr, int E, int expert_offset, int* seg_offsets, int* tile_expert,
                            int* row_src, int* dst_row, int max_rows, cudaStream_t s) {
  return mb_moe_align_pad(idx, n, n_ptr, E, expert_offset, seg_offsets, tile_expert, row_src, dst_row, max_rows, kPad, 1, s);
}

extern "C" int mb_moe_gather(const void* x, void* x_perm, const int* row_src, const int* seg_offsets, int E, int k, int H,
                             int max_rows, cudaStream_t s) {
  if (max_rows == 0) return 0;
  if (H % 8) return -1;
  const int blocks = (max_rows + 7) / 8;   // a row per warp: 7258 tokens × 8 × 2048 54 → 51 µs, 2163 15.6 → 14.6, 12 075 99 → 96 against 8 CTAs an SM that walk
  return static_cast<int>(launch_pdl(moe_gather_kernel, dim3(blocks), dim3(256), 0, s, reinterpret_cast<const bf16*>(x),
                                     reinterpret_cast<bf16*>(x_perm), row_src, seg_offsets, E, k, H, max_rows));
}

extern "C" int mb_moe_combine(const void* y_perm, const float* w, const int* dst_row, void* out, long long T, int k, int H,
                              int identity_rows, cudaStream_t s) {
  if (T == 0) return 0;
  if (H % 8) return -1;
  const int blocks = T < 148 * 16 ? static_cast<int>(T) : 148 * 16;
  return static_cast<int>(launch_pdl(moe_combine_kernel, dim3(blocks), dim3(256), 0, s, reinterpret_cast<const bf16*>(y_perm), w, dst_row,
                                     reinterpret_cast<bf16*>(out), T, k, H, identity_rows));
}

extern "C" int mb_moe_combine_bwd(const void* dout, const void* y_perm, const float* w, const int* row_src, const int* seg_offsets,
                                  int E, void* dy_perm, float* dw, int k, int H, int max_rows, cudaStream_t s) {
  if (max_rows == 0) return 0;
  if (H % 8) return -1;
  const int blocks = (max_rows + 7) / 8 < 148 * 8 ? (max_rows + 7) / 8 : 148 * 8;
  moe_combine_bwd_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<const bf16*>(dout), reinterpret_cast<const bf16*>(y_perm), w, row_src,
                                                seg_offsets, E, reinterpret_cast<bf16*>(dy_perm), dw, k, H, max_rows);
  return static_cast<int>(cudaGetLastError());
}

// See moe_glu_bwd_kernel.  h1, dh1 [max_rows, 2F], act_w [max_rows, F] (in: dout · W2), w and dw [pairs]; F a multiple of 8, 16-byte aligned.
extern "C" int mb_moe_glu_bwd(const void* h1, void* act_w, void* dh1, const float* w, const int* row_src, const int* seg_offsets, int E, float* dw, int F,
                              int max_rows, cudaStream_t s) {
  if (max_rows == 0) return 0;
  if (F % 8) return -1;
  const int blocks = (max_rows + 7) / 8 < 148 * 8 ? (max_rows + 7) / 8 : 148 * 8;
  moe_glu_bwd_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<const bf16*>(h1), reinterpret_cast<bf16*>(act_w), reinterpret_cast<bf16*>(dh1), w, row_src,
                                            seg_offsets, E, dw, F, max_rows);
  return static_cast<int>(cudaGetLastError());
}

// See moe_combine_norm_kernel: y = rmsnorm(Σ_j w · y_perm rows + residual) · norm_w, res_out the sum; H ≤ 4096 and a multiple of 8, all 16-byte aligned.
extern "C" int mb_moe_combine_norm(const void* y_perm, const float* w, const int* dst_row, const void* residual, const void* norm_w, void* y, void* res_out,
                                   long long T, int k, int H, float eps, cudaStream_t s) {
  if (T == 0) return 0;
  if (H <= 0 || H % 8 || H > 4096) return -1;
  if ((reinterpret_cast<uintptr_t>(y_perm) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(norm_w) | reinterpret_cast<uintptr_t>(y) |
       reinterpret_cast<uintptr_t>(res_out)) & 15)
    return -2;
  return static_cast<int>(launch_pdl(moe_combine_norm_kernel, dim3(static_cast<unsigned>(T)), dim3((H / 8 + 63) / 64 * 32), 0, s,
                                     reinterpret_cast<const bf16*>(y_perm), w, dst_row, reinterpret_cast<const bf16*>(residual),
                                     reinterpret_cast<const bf16*>(norm_w), reinterpret_cast<bf16*>(y), reinterpret_cast<bf16*>(res_out), k, H, eps));
}
