// Decode attention of few (request, KV head) segments from the raw projections in one launch (included by paged_decode.cu).
//
// A cluster of `split` CTAs takes a segment.  Every CTA norms and rotates the query heads of the segment's group; warp w of CTA r takes 16-key groups
// 4r + w, 4r + w + 4·split, … with a TMA ring of its own (two groups in flight, no barrier with other warps); the partial results meet in distributed
// shared memory, where CTA r adds up every split-th piece of the output.  The new token's key and value go to the cache from CTA 0; the warp whose
// group holds their slot puts them into its copy of the group, which may have been read before they were written.
//
// What bounds it: the chain of latencies.  Norm + rotation + cache write, splits of a segment and their merge as launches of their own were three such
// chains with a trip through memory between them: 1 request of 1801 tokens, 4 KV heads of 8 query heads each: 2.0 + 9.3 + 2.1 → 10.0 µs;
// 7 requests of 433 to 3001: 1.9 + 12.7 + 2.3 → 13.8.
#pragma once

namespace mbpd {

static constexpr int kDaWarps = 4, kDaStages = 2, kDaKeys = 16, kDaMaxSplit = 16;

struct DecodeAttend {
  const bf16 *q, *k, *v;                 // [batch, heads, D], tokens *_stride apart
  long long q_stride, k_stride, v_stride;
  const bf16 *qw, *kw;                   // norm weights or null
  const int *positions, *block_table, *seq_lens;
  const long long* slots;
  bf16 *kc, *vc, *out;
  int max_blocks, block_size, cache_rows, Hq, Hkv, split;
  float log2_theta, eps, scale;
  int* error_flag;
};

template <int D>
struct DaSmem {
  static constexpr int kHalf = kDaKeys * 128;                      // 64 columns of 16 keys, 128-byte swizzle
  static constexpr int kRows = D / 64 * kHalf;                     // K or V of a group
  static constexpr int kStage = 2 * kRows;
  static constexpr int ring = 0;                                   // [warp][stage]; then [warp][8][D] partial sums
  static constexpr int q = kDaWarps * kDaStages * kStage;          // [8][D + 8] bf16
  static constexpr int o = q + 8 * (D + 8) * 2;                    // [8][D] this CTA's sums
  static constexpr int ml = o + 8 * D * 4;                         // [8] maxima, [8] sums of this CTA; [warp][8] of both
  static constexpr int bars = ml + (16 + 2 * kDaWarps * 8) * 4;
  static constexpr int total = bars + kDaWarps * kDaStages * 8;
};

__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <int D>
__global__ void __launch_bounds__(kDaWarps * 32, 2)
decode_attend_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const DecodeAttend p) {
  using S = DaSmem<D>;
  constexpr int EPL = D / 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(blockIdx.x), hk = static_cast<int>(blockIdx.y), req = static_cast<int>(blockIdx.z);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::bars) + warp * kDaStages;
  bool ok = (mb::smem_u32(smem) & 1023u) == 0;                       // swizzled tiles need 1024-byte alignment
  if (!ok && threadIdx.x == 0) atomicExch(p.error_flag, 64);
  if (lane == 0) {
    for (int i = 0; i < kDaStages; ++i) mb::mbar_init(&full[i], 1);
    mb::mbar_fence_init();
  }
  if (threadIdx.x == 0) {
    mb::tma_prefetch_desc(&tm_k);
    mb::tma_prefetch_desc(&tm_v);
  }
  __syncthreads();
  mb::pdl_trigger();
  mb::pdl_wait();
  const int group = p.Hq / p.Hkv, L = p.seq_lens[req];
  const int groups = (max(L, 0) + kDaKeys - 1) / kDaKeys, first = rank * kDaWarps + warp, step = p.split * kDaWarps;
  const int n = ok && groups > first ? (groups - first + step - 1) / step : 0;      // this warp's groups
  const float pos = static_cast<float>(p.positions[req]);
  long long slot = p.slots[req];
  if (slot >= 0 && !mb::dbg::in_bounds(mb::dbg::kKvSlots, slot, 101)) slot = -1;    // debug build: a slot outside the cache is recorded, not written
  const int* bt = p.block_table + static_cast<long long>(req) * p.max_blocks;
  auto row_of = [&](int i) {                                          // first cache row of this warp's group i
    if (i >= n) return 0;
    const int key = (first + i * step) * kDaKeys;
    const long long blk = bt[key / p.block_size];
    return mb::dbg::in_bounds(mb::dbg::kKvBlocks, blk, 301) ? static_cast<int>(blk) * p.block_size + key % p.block_size : p.cache_rows;   // past the end: zeros
  };
  int rows = row_of(lane), ahead = row_of(32 + lane);                 // lane l: group l of the 32 at hand, of the next 32
  uint8_t* ring = smem + warp * kDaStages * S::kStage;
  auto request = [&](int i, int at) {                                 // group i into stage i mod kDaStages while group `at` is at hand
    const int r = __shfl_sync(0xffffffffu, (i >> 5) == (at >> 5) ? rows : ahead, i & 31);
    if (lane == 0) {
      uint64_t* bar = &full[i % kDaStages];
      uint8_t* to = ring + i % kDaStages * S::kStage;
      mb::mbar_expect_tx(bar, S::kStage);
#pragma unroll
      for (int h = 0; h < D / 64; ++h) {
        mb::tma_load_2d(to + h * S::kHalf, &tm_k, bar, hk * D + h * 64, r);
        mb::tma_load_2d(to + S::kRows + h * S::kHalf, &tm_v, bar, hk * D + h * 64, r);
      }
    }
  };
  for (int i = 0; i < min(n, kDaStages); ++i) request(i, 0);
  // the group's query heads, two per warp
  bf16* sQ = reinterpret_cast<bf16*>(smem + S::q);
  for (int h = warp; h < group; h += kDaWarps) {
    bf16 o1[EPL], o2[EPL];
    mb::norm_rope_values<D>(p.q + req * p.q_stride + static_cast<long long>(hk * group + h) * D, p.qw, pos, p.log2_theta, p.eps, nullptr, lane, o1, o2);
#pragma unroll
    for (int e = 0; e < EPL; ++e) {
      sQ[h * (D + 8) + lane * EPL + e] = o1[e];
      sQ[h * (D + 8) + D / 2 + lane * EPL + e] = o2[e];
    }
  }
  const bf16 *k_new = p.k + req * p.k_stride + static_cast<long long>(hk) * D, *v_new = p.v + req * p.v_stride + static_cast<long long>(hk) * D;
  if (rank == 0 && warp == kDaWarps - 1 && slot >= 0) {
    bf16 o1[EPL], o2[EPL];
    mb::norm_rope_values<D>(k_new, p.kw, pos, p.log2_theta, p.eps, nullptr, lane, o1, o2);
    bf16 *kd = p.kc + (slot * p.Hkv + hk) * D, *vd = p.vc + (slot * p.Hkv + hk) * D;
#pragma unroll
    for (int e = 0; e < EPL; ++e) {
      kd[lane * EPL + e] = o1[e];
      kd[D / 2 + lane * EPL + e] = o2[e];
      vd[lane * EPL + e] = v_new[lane * EPL + e];
      vd[D / 2 + lane * EPL + e] = v_new[D / 2 + lane * EPL + e];
    }
  }
  __syncthreads();
  uint32_t qa[D / 16][2];                                             // A operand: rows 0..7 are the group's heads, 8..15 zero
  {
    const int g = lane >> 2;
    const bf16* qr = sQ + g * (D + 8) + (lane & 3) * 2;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      qa[ks][0] = g < group ? *reinterpret_cast<const uint32_t*>(qr + ks * 16) : 0u;
      qa[ks][1] = g < group ? *reinterpret_cast<const uint32_t*>(qr + ks * 16 + 8) : 0u;
    }
  }
  float o_acc[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;
  float m_i = -INFINITY, l_i = 0.f;                                   // row lane / 4
  const float sl2 = p.scale * kLog2e;
  auto unit16 = [](uint8_t* base, int row, int chunk) {               // 16-byte unit `chunk` of a row, atoms of 64 columns, 128-byte swizzle
    return base + (chunk >> 3) * S::kHalf + row * 128 + (((chunk & 7) ^ (row & 7)) << 4);
  };
  for (int i = 0; i < n; ++i) {
    ok = __all_sync(0xffffffffu, ok && mb::mbar_wait(&full[i % kDaStages], (i / kDaStages) & 1));
    if (!ok) break;
    if (i > 0 && (i & 31) == 0) {
      rows = ahead;
      ahead = row_of(i + 32 + lane);
    }
    uint8_t* sK = ring + i % kDaStages * S::kStage;
    uint8_t* sV = sK + S::kRows;
    const int key0 = (first + i * step) * kDaKeys, r0 = __shfl_sync(0xffffffffu, rows, i & 31);
    bool wrote = false;
    if (slot >= r0 && slot < r0 + kDaKeys) {                          // the new token is in this group
      const int row = static_cast<int>(slot) - r0;
      bf16 o1[EPL], o2[EPL];
      mb::norm_rope_values<D>(k_new, p.kw, pos, p.log2_theta, p.eps, nullptr, lane, o1, o2);
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        const int c1 = lane * EPL + e, c2 = D / 2 + c1;
        reinterpret_cast<bf16*>(unit16(sK, row, c1 >> 3))[c1 & 7] = o1[e];
        reinterpret_cast<bf16*>(unit16(sK, row, c2 >> 3))[c2 & 7] = o2[e];
        reinterpret_cast<bf16*>(unit16(sV, row, c1 >> 3))[c1 & 7] = v_new[c1];
        reinterpret_cast<bf16*>(unit16(sV, row, c2 >> 3))[c2 & 7] = v_new[c2];
      }
      wrote = true;
    }
    if (key0 + kDaKeys > L) {                                         // rows behind the sequence: weight 0, but whatever the page holds may be no number
      for (int u = lane; u < kDaKeys * (D / 8); u += 32) {
        const int row = u / (D / 8);
        if (key0 + row >= L) *reinterpret_cast<uint4*>(unit16(sV, row, u % (D / 8))) = make_uint4(0, 0, 0, 0);
      }
      wrote = true;
    }
    if (wrote) {
      mb::fence_proxy_async();                                        // … before the next group is copied over it
      __syncwarp();
    }
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      uint32_t b[4];
      ldsm_x4(s_addr(unit16(sK, (lane & 7) + ((lane >> 4) << 3), ks * 2 + ((lane >> 3) & 1))), b[0], b[1], b[2], b[3]);
      const uint32_t a[4] = {qa[ks][0], 0u, qa[ks][1], 0u};
      mma16816(s[0], a, b[0], b[1]);
      mma16816(s[1], a, b[2], b[3]);
    }
    float mx = m_i;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (key0 + nt * 8 + (lane & 3) * 2 + e >= L) s[nt][e] = -INFINITY;
        mx = fmaxf(mx, s[nt][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float msc = (mx == -INFINITY) ? 0.f : mx * sl2;
    const float alpha = (m_i == -INFINITY) ? 0.f : exp2f(m_i * sl2 - msc);
    m_i = mx;
    float rs = 0.f;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[nt][e] = exp2f(s[nt][e] * sl2 - msc);
        rs += s[nt][e];
      }
    l_i = l_i * alpha + rs;
#pragma unroll
    for (int c = 0; c < D / 8; ++c) { o_acc[c][0] *= alpha; o_acc[c][1] *= alpha; }
    const uint32_t pa[4] = {pack2(s[0][0], s[0][1]), 0u, pack2(s[1][0], s[1][1]), 0u};
#pragma unroll
    for (int nc = 0; nc < D / 16; ++nc) {
      uint32_t b[4];
      ldsm_x4_t(s_addr(unit16(sV, (lane & 7) + (((lane >> 3) & 1) << 3), nc * 2 + (lane >> 4))), b[0], b[1], b[2], b[3]);
      mma16816(o_acc[2 * nc], pa, b[0], b[1]);
      mma16816(o_acc[2 * nc + 1], pa, b[2], b[3]);
    }
    __syncwarp();
    if (i + kDaStages < n) request(i + kDaStages, i);
  }
  // the four warps' sums, each in its own (now idle) part of the ring
  if (!ok && lane == 0) atomicExch(p.error_flag, 65);
  float* sML = reinterpret_cast<float*>(smem + S::ml);                // [8], [8], then [warp][8] and [warp][8]
  float *wM = sML + 16, *wL = wM + kDaWarps * 8;
  float* sO = reinterpret_cast<float*>(smem + S::o);
  l_i += __shfl_xor_sync(0xffffffffu, l_i, 1);
  l_i += __shfl_xor_sync(0xffffffffu, l_i, 2);
  const int r = lane >> 2;
  if ((lane & 3) == 0) { wM[warp * 8 + r] = m_i; wL[warp * 8 + r] = l_i; }
  float* mine = reinterpret_cast<float*>(ring);
#pragma unroll
  for (int c = 0; c < D / 8; ++c) *reinterpret_cast<float2*>(&mine[r * D + c * 8 + (lane & 3) * 2]) = make_float2(o_acc[c][0], o_acc[c][1]);
  __syncthreads();
  for (int u = threadIdx.x; u < group * (D / 4); u += kDaWarps * 32) {
    const int g = u / (D / 4), d = u % (D / 4) * 4;
    float mm = -INFINITY, ll = 0.f;
    float4 oo = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kDaWarps; ++w) mm = fmaxf(mm, wM[w * 8 + g]);
#pragma unroll
    for (int w = 0; w < kDaWarps; ++w) {
      const float mw = wM[w * 8 + g], a = (mw == -INFINITY) ? 0.f : exp2f((mw - mm) * sl2);
      const float4 x = *reinterpret_cast<const float4*>(smem + w * kDaStages * S::kStage + (g * D + d) * 4);
      ll += wL[w * 8 + g] * a;
      oo.x += x.x * a; oo.y += x.y * a; oo.z += x.z * a; oo.w += x.w * a;
    }
    *reinterpret_cast<float4*>(&sO[g * D + d]) = oo;
    if (d == 0) { sML[g] = mm; sML[8 + g] = ll; }
  }
  mb::cluster_sync();
  // every split-th piece of the output, over the CTAs of the cluster in order
  for (int u = rank + p.split * static_cast<int>(threadIdx.x); u < group * (D / 4); u += p.split * kDaWarps * 32) {
    const int g = u / (D / 4), d = u % (D / 4) * 4;
    float m[kDaMaxSplit], l[kDaMaxSplit], mm = -INFINITY, ll = 0.f;
    float4 x[kDaMaxSplit], oo = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < kDaMaxSplit; ++c) {
      if (c < p.split) {
        m[c] = ld_cluster(mb::smem_of_rank(&sML[g], c));
        l[c] = ld_cluster(mb::smem_of_rank(&sML[8 + g], c));
        x[c] = ld_cluster4(mb::smem_of_rank(&sO[g * D + d], c));
      }
    }
#pragma unroll
    for (int c = 0; c < kDaMaxSplit; ++c)
      if (c < p.split) mm = fmaxf(mm, m[c]);
#pragma unroll
    for (int c = 0; c < kDaMaxSplit; ++c) {
      if (c < p.split) {
        const float a = (m[c] == -INFINITY) ? 0.f : exp2f((m[c] - mm) * sl2);
        ll += l[c] * a;
        oo.x += x[c].x * a; oo.y += x[c].y * a; oo.z += x[c].z * a; oo.w += x[c].w * a;
      }
    }
    const float inv = ll > 0.f ? 1.f / ll : 0.f;
    *reinterpret_cast<uint2*>(p.out + (static_cast<long long>(req) * p.Hq + hk * group + g) * D + d) =
        make_uint2(pack2(oo.x * inv, oo.y * inv), pack2(oo.z * inv, oo.w * inv));
  }
  mb::cluster_sync();                                                 // nobody reads this CTA's memory any more
}

}  // namespace mbpd
